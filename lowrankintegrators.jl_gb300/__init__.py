"""GB300-native engine for the per-step hot path of LowRankIntegrators.jl.

Host-side mirror of the reference's public surface (src/primitives.jl,
src/integrators/*.jl): problems, algorithm objects, ``init`` / ``step`` /
``solve`` and the ``SVDLikeRepresentation`` factors.  Every step runs in the
CUDA library ``liblri_gb300.so`` (include/lri.h) on the current CUDA device;
this module only moves factors between host and device and drives the time
loop of src/primitives.jl:68-80.  There is no CPU fallback: without the
library or a CUDA device every call that computes raises.

The reference accepts an arbitrary Julia closure ``F``; the engine accepts a
fixed menu of flow maps (``ZeroOperator``, ``SylvesterTridiagOperator``) and
data streams (``MatrixDataProblem``).  Substeps use a fixed-step explicit
Runge-Kutta scheme (``RK4(nsub)``, ``Euler(nsub)``, ...) in place of the
reference's adaptive Tsit5 default.
"""
from __future__ import annotations

import ctypes as C
import math
from dataclasses import dataclass, field
from typing import Callable, List, Optional, Sequence, Tuple, Union

import numpy as np

from . import _native, _tuning
from ._native import LriError

__all__ = [
    "SVDLikeRepresentation", "TwoFactorRepresentation", "MatrixDEProblem", "MatrixDataProblem",
    "MatrixHybridProblem", "DLRSolution", "DLRIntegrator",
    "UnconventionalAlgorithm", "RankAdaptiveUnconventionalAlgorithm", "ProjectorSplitting", "GreedyIntegrator",
    "PrimalLieTrotter", "DualLieTrotter", "Strang", "SubstepScheme", "Euler", "Heun", "Midpoint", "RK4",
    "ZeroOperator", "SylvesterTridiagOperator", "BurgersOperator", "LocalFlowOperator", "ReactionDiffusionOperator",
    "registered_flows", "Batch", "MixedEnsemble", "init", "step", "solve",
    "solve_ensemble", "core_condition", "History",
    "LriError", "n_steps",
]


# ---------------------------------------------------------------------------
# Factors and problems (src/primitives.jl:13-49; containers from LowRankArithmetic)
# ---------------------------------------------------------------------------

@dataclass
class SVDLikeRepresentation:
    """Y = U S V^T (U n x r, S r x r, V m x r), host arrays in float64."""
    U: np.ndarray
    S: np.ndarray
    V: np.ndarray

    @property
    def rank(self) -> int:
        return self.S.shape[0]

    @property
    def shape(self) -> Tuple[int, int]:
        return (self.U.shape[0], self.V.shape[0])

    def full(self) -> np.ndarray:
        return self.U @ self.S @ self.V.T

    def copy(self) -> "SVDLikeRepresentation":
        return SVDLikeRepresentation(self.U.copy(), self.S.copy(), self.V.copy())


@dataclass
class TwoFactorRepresentation:
    """Y = U Z^T (U n x r orthonormal, Z m x r), host arrays in float64
    (LowRankArithmetic's TwoFactorRepresentation, used by the greedy
    integrator, src/integrators/greedy_integrator.jl:26-32,73-94)."""
    U: np.ndarray
    Z: np.ndarray

    @property
    def rank(self) -> int:
        return self.U.shape[1]

    @property
    def shape(self) -> Tuple[int, int]:
        return (self.U.shape[0], self.Z.shape[0])

    def full(self) -> np.ndarray:
        return self.U @ self.Z.T

    def copy(self) -> "TwoFactorRepresentation":
        return TwoFactorRepresentation(self.U.copy(), self.Z.copy())


class ZeroOperator:
    """F(X, t) = 0."""
    kind = _native.LRI_OP_ZERO


class SylvesterTridiagOperator:
    """F(X, t) = A X + X B^T (+ diag(theta) X), A and B tridiagonal.

    ``A`` and ``B`` are (sub, diag, sup) triples of length n and m
    (``sub[0]`` and ``sup[-1]`` are ignored).  ``theta`` (length n) is folded
    into A's diagonal.
    """
    kind = _native.LRI_OP_SYLVESTER_TRIDIAG

    def __init__(self, A, B, theta=None):
        sub, dia, sup = (np.asarray(x, dtype=np.float64) for x in A)
        if theta is not None:
            dia = dia + np.asarray(theta, dtype=np.float64)
        self.A = (sub, dia, sup)
        self.B = tuple(np.asarray(x, dtype=np.float64) for x in B)

    def packed(self):
        return np.concatenate(self.A), np.concatenate(self.B)


class BurgersOperator:
    """Periodic central-difference Burgers flow map, column j = sample j:

        F(X, t) = (Dxx X) diag(nu) + alpha (Dx X) .* X + beta Dx(X .* X)

    Dxx = tridiag(1, -2, 1) / h^2 and Dx = tridiag(-1, 0, 1) / (2h), both
    periodic over the n grid points (rows).  The reference's smoke test
    (test/data_agnostic_approximation.jl:16-33) is nu = 0.005 for every
    column, alpha = -1, beta = 0; ``nu`` may also be one value per column.
    """
    kind = _native.LRI_OP_BURGERS_PERIODIC

    def __init__(self, h: float, nu, alpha: float = -1.0, beta: float = 0.0):
        self.h = float(h)
        self.nu = np.asarray(nu, dtype=np.float64)
        self.alpha = float(alpha)
        self.beta = float(beta)

    def params(self):
        return (self.h, self.alpha, self.beta)

    def packed_for(self, n: int, m: int):
        nu = np.broadcast_to(self.nu, (m,)) if self.nu.ndim == 0 else self.nu
        if nu.shape != (m,):
            raise ValueError(f"nu has {nu.shape[0]} entries for {m} columns")
        return np.zeros(0), np.array(nu, dtype=np.float64)


class LocalFlowOperator:
    """A flow map compiled into the library (csrc/flows.cuh; the engine's
    stand-in for a user-supplied F, src/integrators/unconventional.jl:2-4,
    51-79): F(Y)_ij = f(Y_{i-1,j}, Y_ij, Y_{i+1,j}, c_j; h, p0, p1), periodic
    along the rows.  ``flow`` is the registered name or id
    (``registered_flows()``), ``c`` one value or one per column."""
    kind = _native.LRI_OP_LOCAL_FLOW

    def __init__(self, flow, h: float, c, p0: float = 0.0, p1: float = 0.0):
        self.flow = flow
        self.h = float(h)
        self.c = np.asarray(c, dtype=np.float64)
        self.p0 = float(p0)
        self.p1 = float(p1)

    def flow_id(self) -> int:
        names = registered_flows()
        if isinstance(self.flow, str):
            if self.flow not in names:
                raise ValueError(f"no flow map named {self.flow!r} in the library ({names})")
            return names.index(self.flow)
        if not 0 <= int(self.flow) < len(names):
            raise ValueError(f"flow id {self.flow} outside the registry ({names})")
        return int(self.flow)

    def params(self):
        return (self.h, self.p0, self.p1)

    def packed_for(self, n: int, m: int):
        c = np.broadcast_to(self.c, (m,)) if self.c.ndim == 0 else self.c
        if c.shape != (m,):
            raise ValueError(f"c has {c.shape[0]} entries for {m} columns")
        return np.zeros(0), np.array(c, dtype=np.float64)


def ReactionDiffusionOperator(h: float, c, p0: float = 0.0, p1: float = 0.0) -> LocalFlowOperator:
    """F(Y) = (Dxx Y) diag(c) + p0 Y + p1 Y.^3, periodic (Allen-Cahn for
    c = eps^2, p0 = 1, p1 = -1): the registered flow "reaction_diffusion"."""
    return LocalFlowOperator("reaction_diffusion", h, c, p0, p1)


def registered_flows() -> List[str]:
    """Names of the flow maps compiled into the library, by id."""
    lib = _native.load()
    return [lib.lri_flow_name(i).decode() for i in range(int(lib.lri_flow_count()))]


@dataclass
class MatrixDEProblem:
    """dX/dt = F(X, t) on tspan, X(t0) ~ u0 (src/primitives.jl:13-17)."""
    f: object
    u0: SVDLikeRepresentation
    tspan: Tuple[float, float]


class MatrixDataProblem:
    """Low-rank tracking of a data stream (src/primitives.jl:23-30): ``y`` is a
    callable t -> A(t) or a list of snapshots (then tspan = (1, len(y)) and
    the step size defaults to 1)."""

    def __init__(self, y, u0: SVDLikeRepresentation, tspan=None):
        self.y = y
        self.u0 = u0
        if tspan is None:
            if callable(y):
                raise ValueError("tspan is required when the data stream is a function")
            tspan = (1, len(y))
        self.tspan = tspan
        self.f = None


class MatrixHybridProblem:
    """Data-informed basis (src/primitives.jl:32-41): y(t) ~ U(t) Z(t)^T with
    the coefficients following dZ/dt = f(Z, U, t) and U refitted to the data.
    ``y`` is a callable t -> snapshot or a list of snapshots, ``u0`` a
    TwoFactorRepresentation.  On the GPU ``f`` is one of the engine's flow
    maps F, meaning f(Z, U, t) = F(U Z^T, t)^T U (the form the reference's
    test uses, test/data_informed_approximation.jl:73)."""

    def __init__(self, y, f, u0: "TwoFactorRepresentation", tspan):
        self.y = y
        self.f = f
        self.u0 = u0
        self.tspan = tspan


@dataclass
class DLRSolution:
    """Solution history (src/primitives.jl:46-49)."""
    Y: List[Optional[SVDLikeRepresentation]]
    t: List[float]


# ---------------------------------------------------------------------------
# Substep schemes and algorithms (src/integrators/*.jl)
# ---------------------------------------------------------------------------

@dataclass(frozen=True)
class SubstepScheme:
    """Fixed-step explicit RK scheme with a sub-diagonal tableau, run ``nsub``
    times per substep interval (stands in for DiffEq's ``Tsit5()``)."""
    name: str
    a: Tuple[float, ...]
    b: Tuple[float, ...]
    c: Tuple[float, ...]
    nsub: int = 1

    def with_nsub(self, nsub: int) -> "SubstepScheme":
        return SubstepScheme(self.name, self.a, self.b, self.c, int(nsub))

    def to_c(self) -> _native.lri_scheme:
        s = _native.lri_scheme()
        s.nstages = len(self.b)
        s.nsub = int(self.nsub)
        for i in range(len(self.b)):
            s.a[i] = self.a[i]
            s.b[i] = self.b[i]
            s.c[i] = self.c[i]
        return s


def Euler(nsub: int = 1) -> SubstepScheme:
    return SubstepScheme("Euler", (0.0,), (1.0,), (0.0,), nsub)


def Heun(nsub: int = 1) -> SubstepScheme:
    return SubstepScheme("Heun", (0.0, 1.0), (0.5, 0.5), (0.0, 1.0), nsub)


def Midpoint(nsub: int = 1) -> SubstepScheme:
    return SubstepScheme("Midpoint", (0.0, 0.5), (0.0, 1.0), (0.0, 0.5), nsub)


def RK4(nsub: int = 1) -> SubstepScheme:
    return SubstepScheme("RK4", (0.0, 0.5, 0.5, 1.0), (1 / 6, 1 / 3, 1 / 3, 1 / 6), (0.0, 0.5, 0.5, 1.0), nsub)


@dataclass
class UnconventionalAlgorithm:
    """BUG integrator (src/integrators/unconventional.jl:13-21)."""
    K_alg: SubstepScheme = field(default_factory=RK4)
    L_alg: Optional[SubstepScheme] = None
    S_alg: Optional[SubstepScheme] = None

    def __post_init__(self):
        self.L_alg = self.L_alg or self.K_alg
        self.S_alg = self.S_alg or self.K_alg


@dataclass
class RankAdaptiveUnconventionalAlgorithm:
    """Rank-adaptive BUG (src/integrators/rank_adaptive_unconventional.jl:15-23).
    ``rmax`` bounds the rank (and sizes the preallocated buffers); ``rmin`` has
    no reference counterpart and defaults to 1."""
    tol: float
    rmax: int = 32
    K_alg: SubstepScheme = field(default_factory=RK4)
    L_alg: Optional[SubstepScheme] = None
    S_alg: Optional[SubstepScheme] = None
    rmin: int = 1

    def __post_init__(self):
        self.L_alg = self.L_alg or self.K_alg
        self.S_alg = self.S_alg or self.K_alg


class PrimalLieTrotter:
    pass


class DualLieTrotter:
    pass


class Strang:
    pass


@dataclass
class ProjectorSplitting:
    """KSL integrator (src/integrators/projector_splitting.jl:27-41)."""
    order: object = field(default_factory=PrimalLieTrotter)
    K_alg: SubstepScheme = field(default_factory=RK4)
    L_alg: Optional[SubstepScheme] = None
    S_alg: Optional[SubstepScheme] = None

    def __post_init__(self):
        self.L_alg = self.L_alg or self.K_alg
        self.S_alg = self.S_alg or self.K_alg


@dataclass
class GreedyIntegrator:
    """Greedy basis fitting (src/integrators/greedy_integrator.jl:17-24):
    every step refits the factors to the snapshot y(t + dt); Z_alg integrates
    the coefficients of a MatrixHybridProblem.  Fixed rank."""
    Z_alg: SubstepScheme = field(default_factory=RK4)

    @property
    def K_alg(self):
        return self.Z_alg

    L_alg = K_alg
    S_alg = K_alg


def _alg_desc(alg, two_factor: bool = False) -> _native.lri_alg_desc:
    d = _native.lri_alg_desc()
    if isinstance(alg, GreedyIntegrator):
        d.kind = _native.LRI_ALG_GREEDY
        d.two_factor = int(bool(two_factor))
    elif isinstance(alg, UnconventionalAlgorithm):
        d.kind = _native.LRI_ALG_BUG
    elif isinstance(alg, RankAdaptiveUnconventionalAlgorithm):
        d.kind = _native.LRI_ALG_RA_BUG
        d.tol = float(alg.tol)
        d.r_min = int(alg.rmin)
    elif isinstance(alg, ProjectorSplitting):
        d.kind = _native.LRI_ALG_KSL
        if isinstance(alg.order, PrimalLieTrotter):
            d.ksl_order = _native.LRI_KSL_PRIMAL
        elif isinstance(alg.order, DualLieTrotter):
            d.ksl_order = _native.LRI_KSL_DUAL
        elif isinstance(alg.order, Strang):
            d.ksl_order = _native.LRI_KSL_STRANG
        else:
            raise TypeError("unknown projector-splitting order")
    else:
        raise TypeError(f"unsupported algorithm {type(alg).__name__}")
    d.K_alg = alg.K_alg.to_c()
    d.L_alg = alg.L_alg.to_c()
    d.S_alg = alg.S_alg.to_c()
    if d.kind != _native.LRI_ALG_RA_BUG:
        d.r_min = 1
    return d


# ---------------------------------------------------------------------------
# Device batch: the handle the C ABI works on
# ---------------------------------------------------------------------------

def _torch():
    import torch
    if not torch.cuda.is_available():
        raise RuntimeError("lri_gb300 needs a CUDA device; there is no CPU fallback")
    return torch


class Batch:
    """A batch of independent DLRA instances advanced together on the GPU.

    Owns the device copies of the packed factors (U, S, V) and operator
    coefficients, and the C handle (workspace, launch order, CUDA graph).
    """

    def __init__(self, n: Sequence[int], m: Sequence[int], r: Sequence[int], alg, op_kind: int,
                 precision: str = "fp64", r_cap: Optional[Sequence[int]] = None,
                 op_params: Optional[Tuple[float, float, float]] = None, two_factor: bool = False):
        torch = _torch()
        self.torch = torch
        self.lib = _native.load()
        if precision not in ("fp64", "fp32", "df"):
            raise ValueError("precision must be 'fp64', 'fp32' or 'df'")
        self.precision = precision
        # 'df' (double-float) batches exchange FP64 buffers at the ABI
        self.dtype = torch.float32 if precision == "fp32" else torch.float64
        self.np_dtype = np.float32 if precision == "fp32" else np.float64
        self.count = len(n)
        self.n = np.asarray(n, dtype=np.int64)
        self.m = np.asarray(m, dtype=np.int64)
        self.r0 = np.asarray(r, dtype=np.int64)
        if r_cap is None:
            r_cap = self.r0
        self.rcap = np.asarray(r_cap, dtype=np.int64)
        self.alg = alg
        self.op_kind = op_kind
        desc = _native.lri_batch_desc()
        desc.dtype = {"fp64": _native.LRI_F64, "fp32": _native.LRI_F32, "df": _native.LRI_DF}[precision]
        desc.op = op_kind
        desc.count = self.count
        I64P = C.POINTER(C.c_int64)
        desc.n = self.n.ctypes.data_as(I64P)
        desc.m = self.m.ctypes.data_as(I64P)
        desc.r = self.r0.ctypes.data_as(I64P)
        desc.r_cap = self.rcap.ctypes.data_as(I64P)
        if op_params is not None:  # Burgers (h, alpha, beta) or a local flow (h, p0, p1, id), shared by the batch
            desc.burgers_h, desc.burgers_alpha, desc.burgers_beta = (float(x) for x in op_params[:3])
            if len(op_params) > 3:
                desc.flow = int(op_params[3])
        self._algd = _alg_desc(alg, two_factor)
        self.two_factor = bool(two_factor)
        self.handle = C.c_void_p()
        _native.check(self.lib.lri_batch_create(C.byref(self.handle), C.byref(desc), C.byref(self._algd)),
                      "lri_batch_create")
        cnt = self.count
        self.offU = np.zeros(cnt, np.int64)
        self.offS = np.zeros(cnt, np.int64)
        self.offV = np.zeros(cnt, np.int64)
        self.offA = np.zeros(cnt, np.int64)
        self.offB = np.zeros(cnt, np.int64)
        tot = np.zeros(5, np.int64)
        _native.check(self.lib.lri_batch_layout(self.handle, *(x.ctypes.data_as(I64P) for x in
                                                               (self.offU, self.offS, self.offV, self.offA,
                                                                self.offB, tot))), "lri_batch_layout")
        self.totals = tot
        dev = torch.device("cuda", torch.cuda.current_device())
        self.device = dev
        # the factors and coefficients share one buffer (parts on 256-byte
        # boundaries): one allocation and one upload
        self._sizes = [max(int(k), 4) for k in tot]
        al = 256 // np.dtype(self.np_dtype).itemsize
        self._starts = [0]
        for k in self._sizes:
            self._starts.append(self._starts[-1] + -(-k // al) * al)
        self._flat = torch.zeros(self._starts[-1], dtype=self.dtype, device=dev)
        self._parts = self._split(self._flat)
        self.U, self.S, self.V, self.opA, self.opB = self._parts
        self._stage = None
        self.offY = None
        self.has_data = op_kind == _native.LRI_OP_DATA or isinstance(alg, GreedyIntegrator)
        if self.has_data:
            self.offY = np.zeros(cnt, np.int64)
            totY = np.zeros(1, np.int64)
            _native.check(self.lib.lri_batch_data_layout(self.handle, self.offY.ctypes.data_as(I64P),
                                                         totY.ctypes.data_as(I64P)), "lri_batch_data_layout")
            self.totY = int(totY[0])
            self.Ynext = torch.zeros(max(self.totY, 4), dtype=self.dtype, device=dev)
        self.bound = False

    # -- helpers -----------------------------------------------------------
    def _stream(self):
        t = self.torch
        # 0.3 us against 2.9 through a Stream object, in every call of a step
        # loop; not a public function, so it may be missing
        raw = getattr(t._C, "_cuda_getCurrentRawStream", None)
        if raw is None:
            return C.c_void_p(t.cuda.current_stream().cuda_stream)
        return C.c_void_p(raw(t.cuda.current_device()))

    def close(self):
        if getattr(self, "handle", None) is not None and self.handle.value:
            self.lib.lri_batch_destroy(self.handle)
            self.handle = C.c_void_p()

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass

    def _split(self, flat):
        return [flat[a:a + k] for a, k in zip(self._starts, self._sizes)]

    def pack_factors(self, factors: Sequence[SVDLikeRepresentation]):
        """Host-side packing of per-instance factors into the flat layout."""
        return self._pack_into(factors, [np.zeros(k, self.np_dtype) for k in self._sizes[:3]])

    def _pack_into(self, factors, parts):
        hU, hS, hV = parts
        for i, Y in enumerate(factors):
            n, m, rc = int(self.n[i]), int(self.m[i]), int(self.rcap[i])
            r = Y.S.shape[0]
            if Y.U.shape != (n, r) or Y.V.shape != (m, r) or r > rc:
                raise ValueError(f"instance {i}: factor shapes do not match the batch")
            for h, off, rows, X in ((hU, self.offU, n, Y.U), (hS, self.offS, rc, Y.S), (hV, self.offV, m, Y.V)):
                h[off[i]:off[i] + rows * rc].reshape((rows, rc), order="F")[:X.shape[0], :r] = X
        return hU, hS, hV

    def upload(self, factors: Sequence[SVDLikeRepresentation], operators=None):
        t = self.torch
        flat = np.zeros(self._starts[-1], self.np_dtype)
        parts = self._split(flat)
        self._pack_into(factors, parts[:3])
        end = self._starts[3]  # the coefficients stay unless there are new ones
        if operators is not None and self.op_kind == _native.LRI_OP_SYLVESTER_TRIDIAG:
            hA, hB = parts[3:]
            for i, op in enumerate(operators):
                a, b = op.packed()
                if len(a) != 3 * self.n[i] or len(b) != 3 * self.m[i]:
                    raise ValueError(f"instance {i}: operator size does not match the batch")
                hA[self.offA[i]:self.offA[i] + len(a)] = a
                hB[self.offB[i]:self.offB[i] + len(b)] = b
            end = self._starts[5]
        mine = (self.U, self.S, self.V, self.opA, self.opB)
        if all(x is y for x, y in zip(mine, self._parts)):
            self._flat[:end].copy_(t.from_numpy(flat[:end]))
        else:  # buffers that the caller put in their place
            for x, part, start in zip(mine, parts, self._starts):
                if start < end:
                    x.zero_()[:part.size].copy_(t.from_numpy(part))
        if operators is not None and self.op_kind in (_native.LRI_OP_BURGERS_PERIODIC, _native.LRI_OP_LOCAL_FLOW):
            hB = np.zeros(int(self.opB.numel()), self.np_dtype)
            for i, op in enumerate(operators):
                _, b = op.packed_for(int(self.n[i]), int(self.m[i]))
                hB[self.offB[i]:self.offB[i] + len(b)] = b
            self.opB.copy_(t.from_numpy(hB))
        self.bind()

    def bind(self):
        ptr = lambda x: C.c_void_p(x.data_ptr())
        _native.check(self.lib.lri_batch_bind(self.handle, ptr(self.U), ptr(self.S), ptr(self.V),
                                              ptr(self.opA), ptr(self.opB)), "lri_batch_bind")
        self.bound = True

    def pack_data(self, snapshots: Sequence[np.ndarray]) -> np.ndarray:
        return self._pack_data_into(snapshots, np.zeros(self.totY, self.np_dtype))

    def _pack_data_into(self, snapshots, h):
        end = 0
        for i, Y in enumerate(snapshots):
            n, m = int(self.n[i]), int(self.m[i])
            Y = np.asarray(Y)
            if Y.shape != (n, m):
                raise ValueError(f"instance {i}: snapshot shape {Y.shape} != {(n, m)}")
            end = int(self.offY[i]) + n * m
            h[end - n * m:end].reshape((n, m), order="F")[...] = Y
        h[end:] = 0  # instances without a snapshot (the buffer holds an earlier one)
        return h

    # Snapshots up to this size are staged in page-locked memory (two of them
    # per batch: 240 MB, 117 against 135 ms per step from pageable memory); a
    # host is not asked to lock twice the size of larger ones.
    STAGE_BYTES = 256 << 20

    def _send_data(self, fill):
        """fill(host array) writes a snapshot into one of two page-locked
        buffers in turn; its copy to Ynext is queued behind the steps, so the
        host packs the next snapshot while they run.  Where such memory is not
        to be had, from pageable memory."""
        t = self.torch
        if t.cuda.is_current_stream_capturing():
            raise RuntimeError("snapshots cannot be sent from the host while the stream is being captured")
        if self._stage is None:
            self._stage = self._staging_buffers()
        if not self._stage:
            h = np.zeros(max(self.totY, 4), self.np_dtype)
            fill(h)
            self.Ynext.copy_(t.from_numpy(h))
            return
        self._stage.reverse()
        buf, ev = self._stage[0]
        ev.synchronize()  # this buffer's last copy has left it
        fill(buf.numpy())
        self.Ynext.copy_(buf, non_blocking=True)
        ev.record()

    def _staging_buffers(self):
        t = self.torch
        if self.totY * np.dtype(self.np_dtype).itemsize > self.STAGE_BYTES:
            return []
        try:
            return [(t.zeros(max(self.totY, 4), dtype=self.dtype, pin_memory=True), t.cuda.Event()) for _ in range(2)]
        except RuntimeError:  # no page-locked memory left
            return []

    def data_init(self, snapshots: Sequence[np.ndarray]):
        self._send_data(lambda h: self._pack_data_into(snapshots, h))
        _native.check(self.lib.lri_batch_data_init(self.handle, C.c_void_p(self.Ynext.data_ptr()),
                                                   self._stream()), "lri_batch_data_init")

    def step(self, t: float, dt: float, nsteps: int = 1, next_snapshots=None):
        """step!(integrator, alg, dt), ``nsteps`` times (asynchronous)."""
        yptr = None
        if self.has_data:
            if next_snapshots is None:
                raise ValueError("data problems need the next snapshot")
            if isinstance(next_snapshots, np.ndarray) and next_snapshots.ndim == 1:
                if next_snapshots.size not in (1, self.Ynext.numel()):
                    raise RuntimeError(f"{next_snapshots.size} snapshot values, the batch takes {self.Ynext.numel()}")
                self._send_data(lambda h: np.copyto(h, next_snapshots, casting="unsafe"))
            else:
                self._send_data(lambda h: self._pack_data_into(next_snapshots, h))
            yptr = C.c_void_p(self.Ynext.data_ptr())
        _native.check(self.lib.lri_batch_step(self.handle, float(t), float(dt), int(nsteps), yptr,
                                              self._stream()), "lri_batch_step")

    def prepare(self, dt: float, nsteps: int):
        """Builds the CUDA graph of an nsteps-step call ahead of time."""
        if nsteps > 1 and not self.has_data:
            _native.check(self.lib.lri_batch_prepare(self.handle, float(dt), int(nsteps)), "lri_batch_prepare")

    def set_occupancy(self, ctas_per_sm: int):
        """Register budget of the step kernel: 3 (default) or 2 CTAs per SM."""
        _native.check(self.lib.lri_batch_set_occupancy(self.handle, int(ctas_per_sm)), "lri_batch_set_occupancy")
        self.ctas_per_sm = int(ctas_per_sm)

    def apply_tuning(self, table=None):
        """Takes the tuned register budget of this batch's precision and
        dominant rank bucket (``tuning.json``); returns what was chosen.  It
        acts on the step kernel: double-float BUG batches that run by sides
        take and report it without an effect."""
        ctas, bucket = _tuning.ensemble_occupancy(self.precision, self.n, self.m, self.rcap, table)
        if self.precision != "fp64":
            self.set_occupancy(ctas)
        return {"ctas_per_sm": getattr(self, "ctas_per_sm", 3), "bucket": bucket}

    def launches_per_step(self) -> int:
        return int(self.lib.lri_batch_launches_per_step(self.handle))

    def launches(self, nsteps: int) -> int:
        """Kernel launches of one step(t, dt, nsteps) call: the per-step
        engine launches, plus the double-float write-back once per call."""
        per = self.launches_per_step()
        wb = 3 if self.precision == "df" else 0
        return nsteps * (per - wb) + wb

    def ranks(self) -> np.ndarray:
        out = np.zeros(self.count, np.int64)
        _native.check(self.lib.lri_batch_ranks(self.handle, out.ctypes.data_as(C.POINTER(C.c_int64)),
                                               self._stream()), "lri_batch_ranks")
        return out

    def check_status(self):
        _native.check(self.lib.lri_batch_status(self.handle, self._stream()), "device status")

    def download(self) -> List[SVDLikeRepresentation]:
        ranks = self.ranks()
        return self.unpack(self.U.cpu().numpy(), self.S.cpu().numpy(), self.V.cpu().numpy(), ranks)

    def unpack(self, hU, hS, hV, ranks) -> List[SVDLikeRepresentation]:
        """Per-instance factors from host copies of the packed buffers."""
        hU, hS, hV = (np.asarray(h, dtype=np.float64) for h in (hU, hS, hV))
        out = []
        for i in range(self.count):
            n, m, rc, r = int(self.n[i]), int(self.m[i]), int(self.rcap[i]), int(ranks[i])
            U = hU[self.offU[i]:self.offU[i] + n * rc].reshape((n, rc), order="F")[:, :r].copy()
            S = hS[self.offS[i]:self.offS[i] + rc * rc].reshape((rc, rc), order="F")[:r, :r].copy()
            V = hV[self.offV[i]:self.offV[i] + m * rc].reshape((m, rc), order="F")[:, :r].copy()
            out.append(SVDLikeRepresentation(U, S, V))
        return out


class History:
    """The solution history of a batch (lri_history_*): every record is a
    device copy of the factors into a ring slot and an asynchronous copy of
    the slot to page-locked host memory, so the steps do not wait for the
    transfers (the reference deep-copies after every step, update_sol!,
    src/primitives.jl:82-90)."""

    def __init__(self, batch: Batch, slots: int = 8):
        self.b = batch
        self.lib = batch.lib
        self.torch = batch.torch
        self.handle = C.c_void_p()
        _native.check(self.lib.lri_history_create(C.byref(self.handle), batch.handle, int(slots)),
                      "lri_history_create")
        self.pending = []

    def host_buffers(self):
        """Page-locked host buffers (U, S, V, ranks) sized for one record."""
        t, b = self.torch, self.b
        # one allocation, laid out like the device's ring slot (one transfer)
        es = b.U.element_size()
        k = [x.numel() for x in (b.U, b.S, b.V)]
        flat = t.empty(sum(k) * es + max(b.count, 1) * 4, dtype=t.uint8, pin_memory=True)
        f = flat[:sum(k) * es].view(b.dtype)
        return f[:k[0]], f[k[0]:k[0] + k[1]], f[k[0] + k[1]:], flat[sum(k) * es:].view(t.int32)

    def record(self, host=None) -> int:
        """Queues a copy of the batch's current factors; returns its number.
        host: optional buffers from host_buffers() to copy into (the caller
        reuses them once wait() returned for the record that last used
        them); by default new ones are allocated."""
        b = self.b
        hU, hS, hV, hR = host if host is not None else self.host_buffers()
        seq = C.c_int64(0)
        ptr = lambda x: C.c_void_p(x.data_ptr())
        _native.check(self.lib.lri_history_record(self.handle, ptr(hU), ptr(hS), ptr(hV),
                                                  C.cast(hR.data_ptr(), C.POINTER(C.c_int32)), b._stream(),
                                                  C.byref(seq)), "lri_history_record")
        self.pending.append((seq.value, hU, hS, hV, hR))
        return seq.value

    def wait(self, seq: int):
        """Blocks until record seq is in its host buffers."""
        _native.check(self.lib.lri_history_wait(self.handle, int(seq)), "lri_history_wait")

    def collect(self) -> List[List[SVDLikeRepresentation]]:
        """Waits for every queued record; their per-instance factors, in order."""
        out = []
        for seq, hU, hS, hV, hR in self.pending:
            _native.check(self.lib.lri_history_wait(self.handle, seq), "lri_history_wait")
            n = self.b
            out.append(n.unpack(hU.numpy()[:n.U.numel()], hS.numpy()[:n.S.numel()], hV.numpy()[:n.V.numel()],
                                hR.numpy()[:n.count]))
        self.pending = []
        return out

    def close(self):
        if getattr(self, "handle", None) is not None and self.handle.value:
            self.lib.lri_history_destroy(self.handle)
            self.handle = C.c_void_p()

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


# ---------------------------------------------------------------------------
# init / step / solve (src/primitives.jl:54-104; init at unconventional.jl:109-119)
# ---------------------------------------------------------------------------

@dataclass
class DLRIntegrator:
    """src/primitives.jl:54-63, holding the device batch instead of a cache."""
    u: SVDLikeRepresentation
    t: float
    dt: float
    sol: DLRSolution
    alg: object
    batch: Batch
    prob: object
    iter: int = 0
    _snap: int = 0


def n_steps(tspan, dt) -> int:
    """Iterations of the time loop ``while (tf - t)/T > 1e-8; t += dt``
    (src/primitives.jl:70-74)."""
    t0, tf = tspan
    T = tf - t0
    t = t0
    k = 0
    while (tf - t) / T > 1e-8:
        t += dt
        k += 1
    return k


def _init_sol(dt, t0, tf, u0) -> DLRSolution:
    """src/primitives.jl:92-104."""
    if isinstance(dt, (int, np.integer)) and isinstance(t0, (int, np.integer)):
        steps = list(range(t0, tf + 1, dt))
        return DLRSolution([None] * len(steps), [float(s) for s in steps])
    n = int(math.floor((tf - t0) / dt)) + 1
    return DLRSolution([None] * n, list(np.linspace(t0, tf, n)))


def _op_kind(prob) -> int:
    if isinstance(prob, MatrixDataProblem):
        return _native.LRI_OP_DATA
    f = prob.f
    if isinstance(f, ZeroOperator):
        return _native.LRI_OP_ZERO
    if isinstance(f, SylvesterTridiagOperator):
        return _native.LRI_OP_SYLVESTER_TRIDIAG
    if isinstance(f, BurgersOperator):
        return _native.LRI_OP_BURGERS_PERIODIC
    if isinstance(f, LocalFlowOperator):
        return _native.LRI_OP_LOCAL_FLOW
    raise LriError(2, "flow map is not one of the engine's operators (arbitrary closures are unsupported)")


def _has_data(prob) -> bool:
    return isinstance(prob, (MatrixDataProblem, MatrixHybridProblem))


def _op_params(probs):
    """Batch-wide Burgers parameters (h, alpha, beta), or None."""
    fs = [p.f for p in probs if isinstance(p, (MatrixDEProblem, MatrixHybridProblem))
          and isinstance(p.f, (BurgersOperator, LocalFlowOperator))]
    if not fs:
        return None
    ps = {f.params() + ((f.flow_id(),) if isinstance(f, LocalFlowOperator) else ()) for f in fs}
    if len(ps) != 1:
        raise ValueError("the flow-map instances of one batch must share the flow, h and its two scalars")
    return ps.pop()


def _data_at(prob: MatrixDataProblem, t):
    if callable(prob.y):
        return np.asarray(prob.y(t), dtype=np.float64)
    idx = int(round(t))
    if abs(t - idx) > 1e-12:
        raise TypeError("discrete snapshot data needs an integer time step")
    return np.asarray(prob.y[idx - 1], dtype=np.float64)


def init(prob, alg, dt, precision: str = "fp64") -> DLRIntegrator:
    """init(prob, alg, dt) (unconventional.jl:109-119, greedy_integrator.jl:54-71)."""
    t0, tf = prob.tspan
    if not tf > t0:
        raise AssertionError("Integration in reverse time direction is not supported")
    u0 = prob.u0
    two = isinstance(u0, TwoFactorRepresentation)
    if two and not isinstance(alg, GreedyIntegrator):
        raise TypeError("two-factor (U Z^T) representations are integrated by the GreedyIntegrator")
    if isinstance(prob, MatrixHybridProblem) and not (two and isinstance(alg, GreedyIntegrator)):
        raise TypeError("a MatrixHybridProblem takes a TwoFactorRepresentation and the GreedyIntegrator")
    n = u0.U.shape[0]
    m = (u0.Z if two else u0.V).shape[0]
    r = u0.rank
    rcap = r
    if isinstance(alg, RankAdaptiveUnconventionalAlgorithm):
        rcap = max(r, min(alg.rmax, n // 2, m // 2))
    packed = SVDLikeRepresentation(u0.U, np.eye(r), u0.Z) if two else u0
    b = Batch([n], [m], [r], alg, _op_kind(prob), precision, r_cap=[rcap], op_params=_op_params([prob]),
              two_factor=two)
    b.upload([packed], [prob.f] if isinstance(prob, (MatrixDEProblem, MatrixHybridProblem)) else None)
    if isinstance(prob, MatrixDataProblem) and not isinstance(alg, GreedyIntegrator):
        b.data_init([_data_at(prob, t0)])
    sol = _init_sol(dt, t0, tf, u0)
    sol.Y[0] = u0.copy()
    return DLRIntegrator(u0.copy(), t0, dt, sol, alg, b, prob, 0)


def _download_one(b: "Batch"):
    Y = b.download()[0]
    return TwoFactorRepresentation(Y.U, Y.V) if b.two_factor else Y


def step(integ: DLRIntegrator, alg=None, dt=None, sync_factors: bool = True) -> None:
    """step!(integrator, alg, dt): one step on the device."""
    dt = integ.dt if dt is None else dt
    b = integ.batch
    if _has_data(integ.prob):
        b.step(integ.t, dt, 1, [_data_at(integ.prob, integ.t + dt)])
    else:
        b.step(integ.t, dt, 1)
    integ.t += dt
    integ.iter += 1
    if sync_factors:
        b.check_status()
        integ.u = _download_one(b)


def _update_sol(integ: DLRIntegrator) -> None:
    """src/primitives.jl:82-90."""
    if integ.iter <= len(integ.sol.Y) - 1:
        integ.sol.Y[integ.iter] = integ.u.copy()
        integ.sol.t[integ.iter] = integ.t
    else:
        integ.sol.Y.append(integ.u.copy())
        integ.sol.t.append(integ.t)


def solve(prob, alg, dt=None, precision: str = "fp64", save_everystep: bool = True) -> DLRSolution:
    """solve(prob, alg, dt) (src/primitives.jl:68-80).  With
    ``save_everystep=False`` only the initial and final factors are kept and
    DE problems run all steps as one captured CUDA graph."""
    if dt is None:
        if not isinstance(prob, MatrixDataProblem) or callable(prob.y):
            raise ValueError("If the data is not provided as array, integration stepsize needs to be specified")
        dt = 1
    integ = init(prob, alg, dt, precision)
    T = prob.tspan[1] - prob.tspan[0]
    if not save_everystep and not _has_data(prob):
        k = n_steps(prob.tspan, dt)
        integ.batch.step(integ.t, dt, k)
        for _ in range(k):
            integ.t += dt
        integ.iter = k
        integ.batch.check_status()
        integ.u = _download_one(integ.batch)
        integ.sol.Y = [integ.sol.Y[0], integ.u.copy()]
        integ.sol.t = [integ.sol.t[0], integ.t]
        integ.batch.close()
        return integ.sol
    if save_everystep:
        # the history copies overlap the next steps; unpacked once at the end
        hist = History(integ.batch)
        times = []
        try:
            while (prob.tspan[1] - integ.t) / T > 1e-8:
                step(integ, alg, dt, sync_factors=False)
                hist.record()
                times.append(integ.t)
            integ.batch.check_status()
            for k, (Y, tk) in enumerate(zip(hist.collect(), times)):
                Y = Y[0]
                integ.u = TwoFactorRepresentation(Y.U, Y.V) if integ.batch.two_factor else Y
                integ.iter, integ.t = k + 1, tk
                _update_sol(integ)
        finally:
            hist.close()
    else:
        while (prob.tspan[1] - integ.t) / T > 1e-8:
            step(integ, alg, dt, sync_factors=False)
    if not save_everystep:
        integ.batch.check_status()
        integ.u = _download_one(integ.batch)
        integ.sol.Y = [integ.sol.Y[0], integ.u.copy()]
        integ.sol.t = [integ.sol.t[0], integ.t]
    integ.batch.close()
    return integ.sol


def core_condition(S: np.ndarray) -> float:
    """sigma_max / sigma_min of a core matrix (inf when singular)."""
    s = np.linalg.svd(np.asarray(S, dtype=np.float64), compute_uv=False)
    return float(s[0] / s[-1]) if s[-1] > 0 else float("inf")


# The FP32 form (FP32 panels; basis changes, projections and S-step in
# double-float) keeps a rounding floor of a few 1e-6 relative error over a
# hundred steps, independent of the core's conditioning, until the core's
# smallest singular values approach the FP32 rounding level of the largest:
# the K/L panels mix columns of size sigma_1 into columns of size sigma_r, so
# each step perturbs the small directions by u_32 * kappa(S) relative to
# their size.  Measured on the 4096-instance Lyapunov ensemble (103 steps,
# graded cores kappa = 2^(r-1)): max error <= 5.7e-6 up to kappa = 2^22,
# first failures at 2^23, total loss beyond 2^24 = 1/u_32.  The mixed form
# runs an instance in FP32 while kappa(S0) <= 2^21 (u_32 * kappa <= 1/8),
# else in double-float.
MIXED_KAPPA_MAX = 2.0 ** 21


class MixedEnsemble:
    """An ensemble split by core conditioning into an FP32 batch and a
    double-float batch, stepped concurrently on two CUDA streams."""

    def __init__(self, factors: Sequence[SVDLikeRepresentation], operators, alg, op_kind: int,
                 kappa_max: float = MIXED_KAPPA_MAX, r_cap=None, tuned: bool = True):
        op_params = None
        self.tuning = {}
        if op_kind in (_native.LRI_OP_BURGERS_PERIODIC, _native.LRI_OP_LOCAL_FLOW):
            op_params = _op_params([MatrixDEProblem(f, Y, (0.0, 1.0)) for f, Y in zip(operators, factors)])
        torch = _torch()
        self.torch = torch
        self.count = len(factors)
        kap = np.array([core_condition(Y.S) for Y in factors])
        self.kappa = kap
        self.parts = []
        for prec, sel in (("fp32", np.flatnonzero(kap <= kappa_max)), ("df", np.flatnonzero(kap > kappa_max))):
            if len(sel) == 0:
                continue
            fs = [factors[i] for i in sel]
            ops = None if operators is None else [operators[i] for i in sel]
            rc = None if r_cap is None else [r_cap[i] for i in sel]
            b = Batch([Y.U.shape[0] for Y in fs], [Y.V.shape[0] for Y in fs], [Y.S.shape[0] for Y in fs], alg,
                      op_kind, prec, r_cap=rc, op_params=op_params)
            b.upload(fs, ops)
            self.tuning[prec] = b.apply_tuning() if tuned else {"ctas_per_sm": 3, "bucket": None}
            self.parts.append((prec, sel, b, torch.cuda.Stream()))

    def step(self, t: float, dt: float, nsteps: int = 1):
        torch = self.torch
        cur = torch.cuda.current_stream()
        for _, _, b, st in self.parts:
            st.wait_stream(cur)
            with torch.cuda.stream(st):
                b.step(t, dt, nsteps)
        for _, _, b, st in self.parts:
            cur.wait_stream(st)

    def launches_per_step(self) -> int:
        return sum(int(b.lib.lri_batch_launches_per_step(b.handle)) for _, _, b, _ in self.parts)

    def launches(self, nsteps: int) -> int:
        return sum(b.launches(nsteps) for _, _, b, _ in self.parts)

    def prepare(self, dt: float, nsteps: int):
        for _, _, b, _ in self.parts:
            b.prepare(dt, nsteps)

    def check_status(self):
        for _, _, b, st in self.parts:
            with self.torch.cuda.stream(st):
                b.check_status()

    def download(self) -> List[SVDLikeRepresentation]:
        self.torch.cuda.synchronize()
        out = [None] * self.count
        for _, sel, b, _ in self.parts:
            for i, Y in zip(sel, b.download()):
                out[i] = Y
        return out

    def close(self):
        for _, _, b, _ in self.parts:
            b.close()


def solve_ensemble(probs: Sequence[MatrixDEProblem], alg, dt, precision: str = "mixed"
                   ) -> List[SVDLikeRepresentation]:
    """Advances many independent MatrixDEProblems with the same tspan and
    operator kind together; returns the final factors of each.  precision is
    'fp64', 'fp32', 'df' or 'mixed' (FP32 for well-conditioned cores,
    double-float for the others)."""
    tspan = probs[0].tspan
    kinds = {_op_kind(p) for p in probs}
    if len(kinds) != 1 or any(p.tspan != tspan for p in probs):
        raise ValueError("ensemble members must share tspan and operator kind")
    kind = kinds.pop()
    k = n_steps(tspan, dt)
    if precision == "mixed":
        ens = MixedEnsemble([p.u0 for p in probs], [p.f for p in probs], alg, kind)
        ens.step(tspan[0], dt, k)
        ens.check_status()
        out = ens.download()
        ens.close()
        return out
    n = [p.u0.U.shape[0] for p in probs]
    m = [p.u0.V.shape[0] for p in probs]
    r = [p.u0.S.shape[0] for p in probs]
    b = Batch(n, m, r, alg, kind, precision, op_params=_op_params(probs))
    b.upload([p.u0 for p in probs], [p.f for p in probs])
    b.step(tspan[0], dt, k)
    b.check_status()
    out = b.download()
    b.close()
    return out


# ---------------------------------------------------------------------------
# Discrete adjoint of the BUG integrator (no counterpart in the reference)
# ---------------------------------------------------------------------------

def terminal_loss(Y: SVDLikeRepresentation, target):
    """L = ||U S V^T - X_t||_F^2 and its gradient with respect to U, S, V;
    ``target`` is an SVDLikeRepresentation (never formed as n x m) or a dense
    array."""
    U, S, V = Y.U, Y.S, Y.V
    if isinstance(target, SVDLikeRepresentation):
        Wt, Qt = target.U @ target.S, target.V       # X_t = Wt Qt^T
    else:
        Wt, Qt = np.asarray(target, dtype=np.float64), np.eye(V.shape[0])
    VtV, UtU = V.T @ V, U.T @ U
    QtV, WtU = Qt.T @ V, Wt.T @ U
    loss = (np.trace(S.T @ UtU @ S @ VtV) - 2.0 * np.trace(S.T @ WtU.T @ QtV)
            + np.sum((Wt.T @ Wt) * (Qt.T @ Qt)))
    Ub = 2.0 * (U @ S @ VtV @ S.T - Wt @ QtV @ S.T)
    Sb = 2.0 * (UtU @ S @ VtV - WtU.T @ QtV)
    Vb = 2.0 * (V @ S.T @ UtU @ S - Qt @ WtU @ S)
    return float(loss), Ub, Sb, Vb


def bug_gradient(prob: MatrixDEProblem, alg: UnconventionalAlgorithm, dt: float, target,
                 checkpoint_every: int = 20):
    """Loss ||Y(T) - X_t||_F^2 of the BUG solution of ``prob`` (a
    SylvesterTridiagOperator flow, FP64, fixed rank) and its gradient with
    respect to the diagonal of the operator's A (i.e. theta of
    A0 + diag(theta)) and the initial factors.

    The forward run keeps the factors every ``checkpoint_every`` steps on the
    device; the reverse sweep replays each segment once, keeping every
    step's input factors, and runs lri_batch_adjoint_step back through it.
    Returns (loss, theta_bar (n,), SVDLikeRepresentation(U0_bar, S0_bar, V0_bar)).
    """
    if not isinstance(alg, UnconventionalAlgorithm) or not isinstance(prob.f, SylvesterTridiagOperator):
        raise LriError(2, "the adjoint covers BUG on the Sylvester tridiagonal flow")
    torch = _torch()
    u0 = prob.u0
    n, m, r = u0.U.shape[0], u0.V.shape[0], u0.S.shape[0]
    b = Batch([n], [m], [r], alg, _native.LRI_OP_SYLVESTER_TRIDIAG, "fp64")
    try:
        b.upload([u0], [prob.f])
        t0 = prob.tspan[0]
        k = n_steps(prob.tspan, dt)
        c = max(1, int(checkpoint_every))
        ckpts = []
        done = 0
        while done < k:
            ckpts.append((b.U.clone(), b.S.clone(), b.V.clone()))
            seg = min(c, k - done)
            b.step(t0 + done * dt, dt, seg)
            done += seg
        b.check_status()
        _native.check(b.lib.lri_batch_adjoint_prepare(b.handle), "lri_batch_adjoint_prepare")
        loss, Ub, Sb, Vb = terminal_loss(b.download()[0], target)
        dev = b.device
        col = lambda X: torch.from_numpy(np.asarray(X, dtype=np.float64).ravel(order="F")).to(dev)
        Ubar, Sbar, Vbar = col(Ub), col(Sb), col(Vb)
        thb = torch.zeros(n, dtype=torch.float64, device=dev)
        ptr = lambda x: C.c_void_p(x.data_ptr())
        # The replay of a segment depends only on its checkpoint, so segment
        # ci - 1 is replayed on the current stream while the reverse steps of
        # segment ci run on a side stream (the reverse step has its own
        # workspace and reads the replayed inputs only).  The host keeps at
        # most two segments ahead of the reverse sweep, so the saved inputs
        # stay O(checkpoint_every) steps.
        main = torch.cuda.current_stream()
        side = torch.cuda.Stream(device=dev)
        side.wait_stream(main)
        side_ptr = C.c_void_p(side.cuda_stream)
        swept = {}  # segment -> event recorded after its reverse steps

        def replay(ci):
            k0, k1 = ci * c, min(k, ci * c + c)
            if ci + 2 in swept:
                swept.pop(ci + 2).synchronize()
            for dst, src in zip((b.U, b.S, b.V), ckpts[ci]):
                dst.copy_(src)
            b.bind()  # the cached projections belong to the checkpoint's bases
            inputs = []
            for j in range(k0, k1):
                inputs.append((b.U.clone(), b.S.clone(), b.V.clone()))
                b.step(t0 + j * dt, dt, 1)
            ready = torch.cuda.Event()
            ready.record(main)
            return inputs, ready

        nxt = replay(len(ckpts) - 1)
        for ci in reversed(range(len(ckpts))):
            inputs, ready = nxt
            side.wait_event(ready)
            for (U0, S0, V0) in reversed(inputs):
                for x in (U0, S0, V0):
                    x.record_stream(side)
                _native.check(b.lib.lri_batch_adjoint_step(b.handle, float(dt), ptr(U0), ptr(S0), ptr(V0),
                                                           ptr(Ubar), ptr(Sbar), ptr(Vbar), ptr(thb), side_ptr),
                              "lri_batch_adjoint_step")
            ev = torch.cuda.Event()
            ev.record(side)
            swept[ci] = ev
            del inputs
            nxt = replay(ci - 1) if ci > 0 else None
        main.wait_stream(side)
        b.check_status()
        grads = SVDLikeRepresentation(Ubar.cpu().numpy().reshape((r, n)).T.copy(),
                                      Sbar.cpu().numpy().reshape((r, r)).T.copy(),
                                      Vbar.cpu().numpy().reshape((r, m)).T.copy())
        return loss, thb.cpu().numpy(), grads
    finally:
        b.close()


# ---------------------------------------------------------------------------
# One large data stream on the whole GPU (lri_stream_*)
# ---------------------------------------------------------------------------

class DataStreamEngine:
    """Rank-adaptive BUG for one MatrixDataProblem too large for the
    one-CTA-per-instance batch: multi-CTA streaming passes over each pair of
    snapshots (see lri_stream_create).  Snapshots are device tensors holding
    n x m column-major data (``to_device`` converts a host array)."""

    def __init__(self, n: int, m: int, r0: int, rmax: int, tol: float, rmin: int = 1, precision: str = "fp32"):
        torch = _torch()
        self.torch = torch
        self.lib = _native.load()
        if precision not in ("fp32", "fp64"):
            raise ValueError("precision must be 'fp32' or 'fp64'")
        self.dtype = torch.float32 if precision == "fp32" else torch.float64
        self.np_dtype = np.float32 if precision == "fp32" else np.float64
        self.n, self.m, self.R = int(n), int(m), int(rmax)
        self.handle = C.c_void_p()
        code = _native.LRI_F32 if precision == "fp32" else _native.LRI_F64
        _native.check(self.lib.lri_stream_create(C.byref(self.handle), code, self.n, self.m, int(r0), self.R,
                                                 float(tol), int(rmin)), "lri_stream_create")
        dev = torch.device("cuda", torch.cuda.current_device())
        self.device = dev
        self.tuning = None
        if type(self) is DataStreamEngine and self.uses_tensor_cores():
            sr, sc, st, key = _tuning.stream_pass_tiles(self.n, self.m, self.R)
            if key is not None:
                self.set_pass_tiles(sr, sc, st)
                self.tuning = {"shape": key, "splits_rows": sr, "splits_cols": sc, "stages": st}
        self.U = torch.zeros(self.n * self.R, dtype=self.dtype, device=dev)
        self.S = torch.zeros(self.R * self.R, dtype=self.dtype, device=dev)
        self.V = torch.zeros(self.m * self.R, dtype=self.dtype, device=dev)

    def to_device(self, A: np.ndarray):
        A = np.asarray(A)
        if A.shape != (self.n, self.m):
            raise ValueError(f"snapshot shape {A.shape} != {(self.n, self.m)}")
        return self.torch.from_numpy(np.asarray(A, dtype=self.np_dtype).ravel(order="F")).to(self.device)

    def bind(self, Y0: SVDLikeRepresentation):
        r = Y0.S.shape[0]
        u = np.zeros((self.n, self.R), self.np_dtype)
        s = np.zeros((self.R, self.R), self.np_dtype)
        v = np.zeros((self.m, self.R), self.np_dtype)
        u[:, :r], s[:r, :r], v[:, :r] = Y0.U, Y0.S, Y0.V
        for dst, x in ((self.U, u), (self.S, s), (self.V, v)):
            dst.copy_(self.torch.from_numpy(x.ravel(order="F")))
        ptr = lambda x: C.c_void_p(x.data_ptr())
        _native.check(self.lib.lri_stream_bind(self.handle, ptr(self.U), ptr(self.S), ptr(self.V)), "lri_stream_bind")

    def _stream(self):
        return C.c_void_p(self.torch.cuda.current_stream().cuda_stream)

    def step(self, A_prev, A_next):
        _native.check(self.lib.lri_stream_step(self.handle, C.c_void_p(A_prev.data_ptr()),
                                               C.c_void_p(A_next.data_ptr()), self._stream()), "lri_stream_step")

    def greedy_step(self, A_next):
        """GreedyIntegrator step to the snapshot A_next (fixed rank)."""
        _native.check(self.lib.lri_stream_greedy_step(self.handle, C.c_void_p(A_next.data_ptr()), self._stream()),
                      "lri_stream_greedy_step")

    def set_tensor_cores(self, enable: bool):
        """Selects the tensor-core (3xTF32) or CUDA-core snapshot passes."""
        _native.check(self.lib.lri_stream_set_tensor_cores(self.handle, int(bool(enable))),
                      "lri_stream_set_tensor_cores")

    def set_pass_tiles(self, splits_rows: int = 0, splits_cols: int = 0, stages: int = 0):
        """Tile choices of the tensor-core passes (0 = automatic)."""
        _native.check(self.lib.lri_stream_set_pass_tiles(self.handle, int(splits_rows), int(splits_cols), int(stages)),
                      "lri_stream_set_pass_tiles")

    def uses_tensor_cores(self) -> bool:
        v = C.c_int32(0)
        _native.check(self.lib.lri_stream_uses_tensor_cores(self.handle, C.byref(v)), "lri_stream_uses_tensor_cores")
        return bool(v.value)

    def data_product(self, A_prev, A_next, X, trans: bool = False, out=None):
        """(A_next - A_prev) @ X, or its transpose times X, with the stream's
        passes; A_* are device snapshots (see to_device), X a device tensor
        holding a column-major panel (rows x ncols, ncols <= rmax)."""
        rows_x = self.n if trans else self.m
        rows_o = self.m if trans else self.n
        ncols = int(X.numel()) // rows_x
        if out is None:
            out = self.torch.empty(rows_o * self.R, dtype=self.dtype, device=self.device)
        _native.check(self.lib.lri_stream_data_product(self.handle, int(bool(trans)), C.c_void_p(A_prev.data_ptr()),
                                                        C.c_void_p(A_next.data_ptr()), C.c_void_p(X.data_ptr()),
                                                        rows_x, ncols, C.c_void_p(out.data_ptr()), rows_o,
                                                        self._stream()), "lri_stream_data_product")
        return out

    def rank(self) -> int:
        r = C.c_int64(0)
        _native.check(self.lib.lri_stream_rank(self.handle, C.byref(r), self._stream()), "lri_stream_rank")
        return int(r.value)

    def check_status(self):
        _native.check(self.lib.lri_stream_status(self.handle, self._stream()), "stream status")

    def download(self) -> SVDLikeRepresentation:
        r = self.rank()
        U = self.U.cpu().numpy().astype(np.float64).reshape((self.R, self.n)).T[:, :r].copy()
        S = self.S.cpu().numpy().astype(np.float64).reshape((self.R, self.R)).T[:r, :r].copy()
        V = self.V.cpu().numpy().astype(np.float64).reshape((self.R, self.m)).T[:, :r].copy()
        return SVDLikeRepresentation(U, S, V)

    def close(self):
        if getattr(self, "handle", None) is not None and self.handle.value:
            self.lib.lri_stream_destroy(self.handle)
            self.handle = C.c_void_p()

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


def solve_stream(prob: MatrixDataProblem, alg, precision: str = "fp32",
                 save_everystep: bool = True) -> DLRSolution:
    """solve(prob, alg) (src/primitives.jl:68-80) for a MatrixDataProblem given
    as a list of snapshots, on the large-stream engine: rank-adaptive BUG,
    one step per consecutive pair of snapshots, or the GreedyIntegrator
    (fixed rank, one refit per snapshot)."""
    if callable(prob.y):
        raise ValueError("the stream engine takes a list of snapshots")
    u0 = prob.u0
    n, m = u0.U.shape[0], u0.V.shape[0]
    greedy = isinstance(alg, GreedyIntegrator)
    if greedy:
        eng = DataStreamEngine(n, m, u0.S.shape[0], u0.S.shape[0], 0.0, 1, precision)
    else:
        eng = DataStreamEngine(n, m, u0.S.shape[0], min(alg.rmax, 96), alg.tol, alg.rmin, precision)
    try:
        eng.bind(u0)
        sol = DLRSolution([u0.copy()], [float(prob.tspan[0])])
        prev = eng.to_device(prob.y[0])
        for k in range(1, len(prob.y)):
            nxt = eng.to_device(prob.y[k])
            if greedy:
                eng.greedy_step(nxt)
            else:
                eng.step(prev, nxt)
            prev = nxt
            if save_everystep:
                eng.check_status()
                sol.Y.append(eng.download())
                sol.t.append(float(prob.tspan[0] + k))
        eng.check_status()
        if not save_everystep:
            sol.Y.append(eng.download())
            sol.t.append(float(prob.tspan[0] + len(prob.y) - 1))
        return sol
    finally:
        eng.close()


class BurgersLargeEngine(DataStreamEngine):
    """Rank-adaptive BUG for one large BurgersOperator instance (the
    Burgers-UQ workload) on the whole GPU (lri_burgers_*): every flow
    evaluation is a grid of shared-memory tiles of K V^T, never the n x m
    matrix."""

    def __init__(self, op: "BurgersOperator", n: int, m: int, r0: int, rmax: int, tol: float, scheme,
                 rmin: int = 1, precision: str = "fp32"):
        torch = _torch()
        self.torch = torch
        self.lib = _native.load()
        if precision not in ("fp32", "fp64"):
            raise ValueError("precision must be 'fp32' or 'fp64'")
        self.dtype = torch.float32 if precision == "fp32" else torch.float64
        self.np_dtype = np.float32 if precision == "fp32" else np.float64
        self.n, self.m, self.R = int(n), int(m), int(rmax)
        self.handle = C.c_void_p()
        code = _native.LRI_F32 if precision == "fp32" else _native.LRI_F64
        self._sch = scheme.to_c()
        _native.check(self.lib.lri_burgers_create(C.byref(self.handle), code, self.n, self.m, int(r0), self.R,
                                                  float(tol), int(rmin), op.h, op.alpha, op.beta,
                                                  C.byref(self._sch)), "lri_burgers_create")
        dev = torch.device("cuda", torch.cuda.current_device())
        self.device = dev
        self.U = torch.zeros(self.n * self.R, dtype=self.dtype, device=dev)
        self.S = torch.zeros(self.R * self.R, dtype=self.dtype, device=dev)
        self.V = torch.zeros(self.m * self.R, dtype=self.dtype, device=dev)
        _, nu = op.packed_for(self.n, self.m)
        self.nu = torch.from_numpy(np.asarray(nu, dtype=self.np_dtype)).to(dev)

    def bind(self, Y0: SVDLikeRepresentation):
        super().bind(Y0)
        ptr = lambda x: C.c_void_p(x.data_ptr())
        _native.check(self.lib.lri_burgers_bind(self.handle, ptr(self.U), ptr(self.S), ptr(self.V), ptr(self.nu)),
                      "lri_burgers_bind")

    def advance(self, dt: float, nsteps: int = 1):
        _native.check(self.lib.lri_burgers_step(self.handle, float(dt), int(nsteps), self._stream()),
                      "lri_burgers_step")


def solve_burgers_large(prob: MatrixDEProblem, alg: RankAdaptiveUnconventionalAlgorithm, dt: float,
                        precision: str = "fp32", save_everystep: bool = False) -> DLRSolution:
    """solve(prob, alg, dt) (src/primitives.jl:68-80) for one BurgersOperator
    instance too large for the batch, on the whole GPU (rank-adaptive BUG)."""
    if not isinstance(prob.f, BurgersOperator):
        raise LriError(2, "the large Burgers engine takes a BurgersOperator problem")
    u0 = prob.u0
    n, m = u0.U.shape[0], u0.V.shape[0]
    eng = BurgersLargeEngine(prob.f, n, m, u0.S.shape[0], min(alg.rmax, 64), alg.tol, alg.K_alg, alg.rmin, precision)
    try:
        eng.bind(u0)
        t0 = prob.tspan[0]
        sol = DLRSolution([u0.copy()], [float(t0)])
        k = n_steps(prob.tspan, dt)
        if save_everystep:
            for j in range(k):
                eng.advance(dt, 1)
                eng.check_status()
                sol.Y.append(eng.download())
                sol.t.append(float(t0 + (j + 1) * dt))
        else:
            eng.advance(dt, k)
            eng.check_status()
            sol.Y.append(eng.download())
            sol.t.append(float(t0 + k * dt))
        return sol
    finally:
        eng.close()
