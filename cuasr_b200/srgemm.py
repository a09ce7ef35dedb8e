"""Host-side mirror of the reference's device-level operators, over the C ABI.

`Srgemm` and `SrgemmSplitKParallel` keep the method names, argument meaning and status codes of
cuasr::gemm::device::Srgemm (include/cuasr/gemm/device/srgemm.h:139-356) and
cuasr::gemm::device::SrgemmSplitKParallel (include/cuasr/gemm/device/srgemm_splitk_parallel.h:155-378);
template parameters become constructor arguments.  Matrices are device pointers with one leading
dimension (cutlass::TensorRef); torch CUDA tensors are accepted wherever a pointer is.
"""
from __future__ import annotations

import ctypes
import dataclasses
import struct
from typing import Any, Optional, Tuple

import numpy as np

from . import _lib
from .semiring import DType, Layout, NUMPY_DTYPE, Op, Status, annihilator, identity


def _ptr(x: Any) -> int:
    """Device address of a tensor or an address; 0 for None."""
    if x is None:
        return 0
    if type(x) is int:
        return x
    data_ptr = getattr(x, "data_ptr", None)
    return int(x) if data_ptr is None else data_ptr()


# One call packs its arguments with a single struct.pack and makes a single call into the library: a 64 x 64 x 64
# product runs for about 5 us on the device, so what the host does per call decides how often it can be made.
_PACK_SCALAR = {DType.F32: struct.Struct("<f4x").pack, DType.F64: struct.Struct("<d").pack,
                DType.S32: struct.Struct("<i4x").pack, DType.U32: struct.Struct("<I4x").pack}
# the layout of _lib.Args
_PACK_ARGS = struct.Struct("4iQqQqQqQq8s8s8s8sQNQ").pack
assert struct.calcsize("4iQqQqQqQq8s8s8s8sQNQ") == ctypes.sizeof(_lib.Args)
_WRAPPED = (ctypes.c_int32, ctypes.c_int64, ctypes.c_size_t, ctypes.c_void_p)
_STATUS = {int(st): st for st in Status}


def _scalar(value, dtype: DType) -> bytes:
    """The element `value` of type `dtype`, in eight bytes: for values _PACK_SCALAR refuses, because the element type
    cannot hold them or they need a conversion first."""
    return np.asarray(value).astype(NUMPY_DTYPE[dtype]).tobytes().ljust(8, b"\0")


def _stream_handle(stream) -> int:
    if stream is None:
        return 0
    if hasattr(stream, "cuda_stream"):
        return int(stream.cuda_stream)
    return int(stream)


@dataclasses.dataclass
class Arguments:
    """device::Srgemm::Arguments (device/srgemm.h:139-183)."""
    problem_size: Tuple[int, int, int]                 # (M, N, K)
    ref_A: Tuple[Any, int]                             # (pointer or tensor, leading dimension)
    ref_B: Tuple[Any, int]
    ref_C: Tuple[Any, int]
    ref_D: Tuple[Any, int]
    epilogue: Tuple[Any, ...] = ()                     # (), (alpha,), or (alpha, beta)
    split_k_slices: int = 1


class _Operator:
    _splitk_parallel = False

    def __init__(self, add_op: Op, mul_op: Op, dtype: DType = DType.F32,
                 layout_a: Layout = Layout.COLUMN_MAJOR, layout_b: Layout = Layout.COLUMN_MAJOR,
                 layout_c: Layout = Layout.COLUMN_MAJOR, split_k_serial: bool = False,
                 add_identity=None, mul_identity=None):
        self.add_op, self.mul_op, self.dtype = Op(add_op), Op(mul_op), DType(dtype)
        self.layout_a, self.layout_b, self.layout_c = Layout(layout_a), Layout(layout_b), Layout(layout_c)
        self.kSplitKSerial = bool(split_k_serial)
        # AdditionOp::Identity / MultiplicationOp::Identity of the functors the operator is "instantiated" with
        self.add_identity = identity(self.add_op, self.dtype) if add_identity is None else add_identity
        self.mul_identity = identity(self.mul_op, self.dtype) if mul_identity is None else mul_identity
        self._lib = _lib.load()
        self._desc = _lib.Desc(int(self.add_op), int(self.mul_op), int(self.dtype), int(self.layout_a),
                               int(self.layout_b), int(self.layout_c), int(self.kSplitKSerial), 0)
        self._pack_scalar = _PACK_SCALAR[self.dtype]
        self._desc_ref = ctypes.byref(self._desc)
        name = "cuasr_b200_srgemm_splitk" if self._splitk_parallel else "cuasr_b200_srgemm"
        self._run_fn = getattr(self._lib, name)
        # EpilogueOutputOp::Params defaults (semiring_linear_combination.h:67-85)
        self._default_beta = annihilator(self.mul_op, self.dtype)
        self._args: Optional[_lib.Args] = None
        self._keepalive = None

    # -- helpers ---------------------------------------------------------------------------------------
    def _pack(self, args: Arguments, workspace=None, workspace_bytes: int = 0, stream=None) -> _lib.Args:
        m, n, k = args.problem_size
        epi = args.epilogue
        alpha = epi[0] if len(epi) >= 1 else self.mul_identity
        beta = epi[1] if len(epi) >= 2 else self._default_beta
        pack = self._pack_scalar
        try:
            alpha, beta, add_identity, mul_identity = pack(alpha), pack(beta), pack(self.add_identity), pack(self.mul_identity)
        except (struct.error, OverflowError, TypeError):
            alpha, beta, add_identity, mul_identity = (_scalar(v, self.dtype) for v in
                                                       (alpha, beta, self.add_identity, self.mul_identity))
        (A, lda), (B, ldb), (C, ldc), (D, ldd) = args.ref_A, args.ref_B, args.ref_C, args.ref_D
        if workspace is not None and workspace_bytes == 0 and hasattr(workspace, "numel"):
            workspace_bytes = workspace.numel() * workspace.element_size()
        fields = (int(m), int(n), int(k), int(args.split_k_slices), _ptr(A), int(lda), _ptr(B), int(ldb), _ptr(C), int(ldc),
                  _ptr(D), int(ldd), alpha, beta, add_identity, mul_identity, _ptr(workspace), int(workspace_bytes),
                  0 if stream is None else _stream_handle(stream))
        try:
            return _lib.Args.from_buffer_copy(_PACK_ARGS(*fields))
        except struct.error:                # a number its C field cannot hold: wrapped around, as ctypes assigns it
            return _lib.Args(*(kind(v).value if kind in _WRAPPED else _lib.Scalar.from_buffer_copy(v)
                               for v, (_, kind) in zip(fields, _lib.Args._fields_)))

    def _fn(self, base: str):
        name = "cuasr_b200_srgemm_splitk" if self._splitk_parallel else "cuasr_b200_srgemm"
        return getattr(self._lib, name + base)

    # -- the reference's interface -----------------------------------------------------------------------
    def can_implement(self, args: Arguments) -> Status:
        return Status(self._fn("_can_implement")(ctypes.byref(self._desc), ctypes.byref(self._pack(args))))

    def get_workspace_size(self, args: Arguments) -> int:
        return int(self._fn("_workspace_size")(ctypes.byref(self._desc), ctypes.byref(self._pack(args))))

    def get_optional_workspace_size(self, args: Arguments) -> int:
        """Bytes of OPTIONAL workspace for an unsplit launch (0 = nothing to gain): it buys a balanced last wave and
        K-contiguous, aligned copies of operands that would otherwise be gathered element by element."""
        return int(self._lib.cuasr_b200_srgemm_optional_workspace_size(ctypes.byref(self._desc),
                                                                      ctypes.byref(self._pack(args))))

    def initialize(self, args: Arguments, workspace=None, stream=None, workspace_bytes: int = 0) -> Status:
        packed = self._pack(args, workspace, workspace_bytes, stream)
        status = Status(self._fn("_can_implement")(ctypes.byref(self._desc), ctypes.byref(packed)))
        if status != Status.kSuccess:
            return status
        need = self._fn("_workspace_size")(ctypes.byref(self._desc), ctypes.byref(packed))
        if need > 0 and packed.workspace is None:
            return Status.kErrorWorkspaceNull
        self._args = packed
        self._keepalive = (args, workspace)
        return Status.kSuccess

    def update(self, args: Arguments, workspace=None, workspace_bytes: int = 0) -> Status:
        """Refreshes pointers only (device/srgemm.h:285-300)."""
        if self._args is None:
            return Status.kErrorInternal
        stream = self._args.stream
        self._args = self._pack(args, workspace, workspace_bytes, stream)
        self._keepalive = (args, workspace)
        return Status.kSuccess

    def run(self, stream=None) -> Status:
        if self._args is None:
            return Status.kErrorInternal
        if stream is not None:
            self._args.stream = _stream_handle(stream)
        return _STATUS[self._run_fn(self._desc_ref, ctypes.byref(self._args))]

    def run_push(self, extra_outputs, stream=None) -> Status:
        """run(), with every element of D also stored to each matrix in `extra_outputs` (pointers or tensors
        with D's layout and leading dimension; peer-GPU memory allowed): cuasr_b200_srgemm_push."""
        if self._args is None or self._splitk_parallel:
            return Status.kErrorInternal
        if stream is not None:
            self._args.stream = _stream_handle(stream)
        ptrs = (ctypes.c_void_p * max(1, len(extra_outputs)))(*[_ptr(x) for x in extra_outputs])
        return Status(self._lib.cuasr_b200_srgemm_push(ctypes.byref(self._desc), ctypes.byref(self._args),
                                                       len(extra_outputs), ptrs))

    def run_screened(self, args: Arguments, pieces: int = 0, workspace=None, stream=None) -> Status:
        """The product on the kernel that screens in 16 bits, whatever the operands: cuasr_b200_srgemm_screened."""
        return Status(self._lib.cuasr_b200_srgemm_screened(ctypes.byref(self._desc),
                                                           ctypes.byref(self._pack(args, workspace, 0, stream)), int(pieces)))

    def __call__(self, args: Optional[Arguments] = None, workspace=None, stream=None,
                 workspace_bytes: int = 0) -> Status:
        if args is None:
            return self.run(stream)
        # initialize + run: the library's run entry point makes every check that initialize() makes
        packed = self._pack(args, workspace, workspace_bytes, stream)
        status = _STATUS[self._run_fn(self._desc_ref, ctypes.byref(packed))]
        if status is Status.kSuccess:
            self._args = packed
            self._keepalive = (args, workspace)
        return status

    # -- extras ------------------------------------------------------------------------------------------
    def last_kernel(self) -> str:
        return self._lib.cuasr_b200_last_kernel().decode()

    def last_route(self) -> str:
        """What the last product call of this thread launched (cuasr_b200_last_route)."""
        return self._lib.cuasr_b200_last_route().decode()


class Srgemm(_Operator):
    """cuasr::gemm::device::Srgemm."""


class SrgemmSplitKParallel(_Operator):
    """cuasr::gemm::device::SrgemmSplitKParallel."""
    _splitk_parallel = True


def srgemm_path(operator: _Operator, problem_size, ref_A, ref_B, ref_dist, ref_parent, k_offset: int = 0,
                stream=None) -> Status:
    """dist <- min/max(dist, A (x) B) in place with the winning contraction index recorded in `parent` (int32, same
    layout as dist): cuasr_b200_srgemm_path.  `operator` supplies ring (min-plus or max-plus), type and layouts."""
    args = Arguments(problem_size, ref_A, ref_B, ref_dist, ref_dist)
    packed = operator._pack(args, None, 0, stream)
    lib = _lib.load()
    return Status(lib.cuasr_b200_srgemm_path(ctypes.byref(operator._desc), ctypes.byref(packed), _ptr(ref_parent[0]),
                                             int(ref_parent[1]), int(k_offset)))


STATIC_SCRATCH_BYTES = 16 * 1024 * 1024 + 4096


def srgemm_splitk_static(operator: _Operator, args: Arguments, stream=None) -> Status:
    """Split-K SRGEMM on the library's built-in static scratch (cuasr_b200_srgemm_splitk_static): for callers
    that are not allowed to allocate device memory.  `operator` supplies the ring, element type and layouts;
    no workspace is passed.  Calls that overlap on the GPU share the scratch and must be serialised."""
    packed = operator._pack(args, None, 0, stream)
    lib = _lib.load()
    return Status(lib.cuasr_b200_srgemm_splitk_static(ctypes.byref(operator._desc), ctypes.byref(packed)))


def pack_k_contiguous(dtype: DType, src, ld_src: int, src_k_contiguous: bool, rows: int, k: int, dst, ld_dst: int,
                      stream=None) -> Status:
    """cuasr_b200_pack_k_contiguous: copies a rows x k operand (tensors or device addresses) into storage that is
    contiguous along k, dst[r * ld_dst + kk], from src[r + kk * ld_src] or (src_k_contiguous) src[r * ld_src + kk].
    A column-major A packed this way is passed on as a row-major A with leading dimension ld_dst."""
    return Status(_lib.load().cuasr_b200_pack_k_contiguous(int(dtype), _ptr(src), int(ld_src), int(bool(src_k_contiguous)),
                                                           int(rows), int(k), _ptr(dst), int(ld_dst),
                                                           _stream_handle(stream)))


def device_status(stream=None) -> int:
    """Synchronises `stream` and returns the device-side status word (0 = ok)."""
    return int(_lib.load().cuasr_b200_device_status(_stream_handle(stream)))


def launch_count() -> int:
    return int(_lib.load().cuasr_b200_launch_count())
