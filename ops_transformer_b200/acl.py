"""Host-side mirror of the reference operator interface on top of the C ABI.

``grouped_matmul_v4`` follows aclnnGroupedMatmulV4 (gmm/grouped_matmul/op_host/op_api/aclnn_grouped_matmul_v4.h:66-86
of the reference) and ``grouped_matmul_swiglu_quant`` follows aclnnGroupedMatmulSwigluQuant
(gmm/grouped_matmul_swiglu_quant/op_host/op_api/aclnn_grouped_matmul_swiglu_quant.h:37-52): same argument
names and meaning, same two-phase sequence (GetWorkspaceSize -> allocate -> launch on a stream), same status
codes raised as ``AclnnError``.  torch is used for device memory and streams only.
"""
from __future__ import annotations

import array
import contextlib
import ctypes as C
import struct
import threading
from typing import Optional, Sequence

import torch

from . import _lib
from ._lib import LaunchOptions  # noqa: F401  (re-exported: the per-call options of include/gmm_b200.h)
from ._lib import (ACL_BF16, ACL_FLOAT, ACL_FLOAT16, ACL_FORMAT_FRACTAL_NZ, ACL_FORMAT_ND, ACL_INT8, ACL_INT32, ACL_INT64,
                   ACLNN_SUCCESS)

_DTYPES = {
    torch.float32: ACL_FLOAT, torch.float16: ACL_FLOAT16, torch.int8: ACL_INT8, torch.int32: ACL_INT32,
    torch.int64: ACL_INT64, torch.bfloat16: ACL_BF16,
}


class AclnnError(RuntimeError):
    """A non-zero aclnnStatus.  ``status`` holds the code, the text comes from aclGetRecentErrMsg."""

    def __init__(self, status: int, where: str):
        self.status = int(status)
        super().__init__(f"{where} failed with aclnnStatus {status}: {_lib.last_error()}")


def _i64(values: Sequence[int]):
    return (C.c_int64 * len(values))(*values)


def create_tensor(t: torch.Tensor, fmt: int = ACL_FORMAT_ND, dtype: Optional[int] = None,
                  view_dims: Optional[Sequence[int]] = None) -> int:
    """aclCreateTensor over a torch tensor's view (dims, strides, device address).  The caller destroys it.
    ``view_dims``: the tensor is the storage (its shape becomes the storage shape) and is viewed with these dimensions,
    as a FRACTAL_NZ weight is: storage [E, N/32, K/16, 16, 32], view [E, K, N]."""
    storage = list(t.shape)
    if view_dims is None:
        dims, strides = storage, list(t.stride())
    else:
        dims = list(view_dims)
        strides = [1] * len(dims)
        for i in range(len(dims) - 2, -1, -1):
            strides[i] = strides[i + 1] * dims[i + 1]
    code = _DTYPES[t.dtype] if dtype is None else dtype
    h = _lib.lib().aclCreateTensor(_i64(dims), len(dims), code, _i64(strides), 0, fmt, _i64(storage), len(storage),
                                   C.c_void_p(t.data_ptr()))
    if not h:
        raise MemoryError("aclCreateTensor returned null")
    return h


def format_cast_nz(weight: torch.Tensor) -> torch.Tensor:
    """int8 [E, K, N] -> the FRACTAL_NZ storage [E, N/32, K/16, 16, 32] (a copy; K % 16 == 0, N % 32 == 0): element
    (k, n) moves to [n // 32, k // 16, k % 16, n % 32].  What a caller of the reference does once per weight with its
    framework's format cast before calling the WeightNZ operators; a set-up step, not part of the hot path."""
    E, K, N = weight.shape
    if K % 16 or N % 32:
        raise ValueError("FRACTAL_NZ needs K % 16 == 0 and N % 32 == 0")
    return weight.reshape(E, K // 16, 16, N // 32, 32).permute(0, 3, 1, 2, 4).contiguous()


def create_tensor_list(tensors: Sequence[torch.Tensor], fmt: int = ACL_FORMAT_ND) -> int:
    """aclCreateTensorList; the list owns its tensor handles (aclDestroyTensorList frees them)."""
    hs = [create_tensor(t, fmt) for t in tensors]
    arr = (C.c_void_p * len(hs))(*hs)
    h = _lib.lib().aclCreateTensorList(arr, len(hs))
    if not h:
        raise MemoryError("aclCreateTensorList returned null")
    return h


class _Slot:
    """The pooled workspace of one stream.  ``lock`` is held while a call is enqueued with ``buf``: the clear and the kernels of
    two calls must not interleave on the stream."""
    __slots__ = ("lock", "buf")

    def __init__(self):
        self.lock = threading.RLock()
        self.buf: Optional[torch.Tensor] = None


class _Workspace:
    """Growing device buffers for the calls that bring no workspace, one per device and stream: a call uses its buffer until
    its last kernel is done, so calls that may run at the same time must not share one.  The buffers are allocated on their
    own stream; one that is outgrown or evicted goes back to the allocator, which reuses it in that stream's order."""
    MAX_SLOTS = 16   # streams with a buffer; with more of them the oldest slot's goes

    def __init__(self):
        self._slots = {}
        self._lock = threading.Lock()
        self._replayed = {}   # address -> buffer a replay will use (see for_capture)

    def slot(self, device: torch.device, handle: int) -> _Slot:
        # the per-thread default stream has one handle and is another stream in every thread
        key = (device.type, device.index, handle, threading.get_ident() if handle == _STREAM_PER_THREAD else 0)
        s = self._slots.get(key)
        if s is None:
            with self._lock:
                s = self._slots.setdefault(key, _Slot())
                while len(self._slots) > self.MAX_SLOTS:
                    del self._slots[next(iter(self._slots))]
        return s

    def lend(self, slot: _Slot, device: torch.device, stream, nbytes: int) -> torch.Tensor:
        """A workspace of at least ``nbytes`` for the call that is about to be enqueued with the slot's lock held."""
        return (self.for_capture if device.type == "cuda" and _capturing(stream) else self.grown)(slot, device, stream, nbytes)

    @staticmethod
    def grown(slot: _Slot, device: torch.device, stream, nbytes: int) -> torch.Tensor:
        """The slot's buffer with room for ``nbytes``."""
        if slot.buf is None or slot.buf.numel() < nbytes:
            with _on_stream(stream, device):
                slot.buf = torch.empty(int(nbytes), dtype=torch.uint8, device=device)
        return slot.buf

    def for_capture(self, slot: _Slot, device: torch.device, stream, nbytes: int) -> torch.Tensor:
        """A workspace for a call that is being captured.  A buffer from the memory pool of a torch graph belongs to that graph
        as long as it lives, so that its replays share it neither with other graphs nor with calls outside.  A capture that
        has no such pool gets the stream's buffer, which is kept from then on even if the stream's calls outgrow it."""
        with _on_stream(stream, device):
            b = torch.empty(int(nbytes), dtype=torch.uint8, device=device)
        if _in_graph_pool(b):
            return b
        b = self.grown(slot, device, stream, nbytes)
        self._replayed[b.data_ptr()] = b
        return b


_WS = _Workspace()
_STREAM_PER_THREAD = 2   # cudaStreamPerThread


def _on_stream(stream, device: torch.device):
    """Context in which torch's current stream is ``stream``."""
    if stream is None or device.type != "cuda":
        return contextlib.nullcontext()
    if not isinstance(stream, torch.cuda.Stream):
        stream = torch.cuda.ExternalStream(int(stream.cuda_stream), device=device)
    return torch.cuda.stream(stream)


def _capturing(stream) -> bool:
    if stream is None:
        return torch.cuda.is_current_stream_capturing()
    return _lib.lib().gmmB200StreamIsCapturing(int(stream.cuda_stream)) != 0


def _in_graph_pool(t: torch.Tensor) -> bool:
    p = t.data_ptr()
    return any(tuple(seg["segment_pool_id"]) != (0, 0) for seg in torch.cuda.memory_snapshot()
               if seg["address"] <= p < seg["address"] + seg["total_size"])


def _with_pooled(device: torch.device, stream, handle: int, nbytes: int, call):
    """``call(workspace)``, which enqueues on ``stream``, with a pooled workspace of ``nbytes``; returns the workspace."""
    slot = _WS.slot(device, handle)
    with slot.lock:
        workspace = _WS.lend(slot, device, stream, nbytes)
        call(workspace)
        return workspace


def _stream_handle(stream) -> int:
    if stream is None:
        stream = torch.cuda.current_stream()
    return int(stream.cuda_stream)


def _gpu_stream_handle(stream) -> int:
    """The same where CUDA is known to be up, without the stream object that torch.cuda.current_stream builds."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice()) if stream is None else int(stream.cuda_stream)


def check_status(workspace: Optional[torch.Tensor], stream=None) -> None:
    """Synchronise the stream and raise if a kernel recorded a problem in the workspace status word."""
    rec = (C.c_int32 * 4)()
    ptr = C.c_void_p(workspace.data_ptr()) if workspace is not None else None
    size = workspace.numel() if workspace is not None else 0
    rc = _lib.lib().gmmB200CheckStatus(ptr, size, C.c_void_p(_stream_handle(stream)), rec)
    if rc != ACLNN_SUCCESS:
        err = AclnnError(rc, "gmmB200CheckStatus")
        err.record = tuple(int(v) for v in rec)   # (code, CTA, waiting role, detail)
        raise err


def _put(words: list, t: Optional[torch.Tensor], fmt: int = ACL_FORMAT_ND, view_dims: Optional[Sequence[int]] = None) -> None:
    """Append one tensor to a packed description (gmmB200Call, include/gmm_b200.h); the same view as ``create_tensor``."""
    words += array.array("q", _lib.describe((t, fmt, view_dims)))


def _ints(values: Optional[Sequence[int]]) -> Optional[list]:
    return None if values is None else list(values)


def _call(op: int, name: str, words, device: torch.device, workspace: Optional[torch.Tensor], stream,
          options: Optional[LaunchOptions]) -> Optional[torch.Tensor]:
    """Both phases of operator ``name`` on the packed description (bytes or a list of its words); returns the workspace that was
    used (None if none)."""
    if not isinstance(words, bytes):
        words = array.array("q", words).tobytes()
    on_gpu = device.type == "cuda"
    handle = _gpu_stream_handle(stream) if on_gpu else 0
    if workspace is not None:
        return _enqueue(op, name, words, device, workspace, stream, handle, options, None)
    slot = _WS.slot(device, handle)
    with slot.lock:
        return _enqueue(op, name, words, device, None, stream, handle, options, slot)


def _enqueue(op: int, name: str, words: bytes, device: torch.device, workspace: Optional[torch.Tensor], stream, handle: int,
             options: Optional[LaunchOptions], slot: Optional[_Slot]) -> Optional[torch.Tensor]:
    L = _lib.lib()
    res = _lib.CallResult()
    # validation needs no device: tensors that are not on one are planned only, so that what is wrong with them is reported first
    on_gpu = device.type == "cuda"
    buf = None if not on_gpu else workspace if slot is None else slot.buf
    rc = L.gmmB200Call(op if slot is None else op | _lib.OP_POOLED, words, len(words) // 8, buf.data_ptr() if buf is not None else None,
                       buf.numel() if buf is not None else 0, C.byref(options) if options is not None else None, handle, C.byref(res))
    if rc == ACLNN_SUCCESS and res.stage == _lib.STAGE_PLANNED:
        ex = C.c_void_p(res.executor)
        if workspace is not None and workspace.numel() < res.workspaceSize:
            L.aclDestroyAclOpExecutor(ex)
            raise ValueError(f"workspace of {workspace.numel()} bytes is smaller than the {res.workspaceSize} required")
        try:
            buf = workspace if slot is None else _WS.lend(slot, device, stream, res.workspaceSize)
            handle = handle if on_gpu else _stream_handle(stream)
        except Exception:
            L.aclDestroyAclOpExecutor(ex)
            raise
        rc = getattr(L, name)(buf.data_ptr(), res.workspaceSize, ex, handle)
        res.stage = _lib.STAGE_RUN
    if rc != ACLNN_SUCCESS:
        raise AclnnError(rc, name + ("GetWorkspaceSize" if res.stage == _lib.STAGE_PLAN else
                                     ": gmmB200SetExecutorOptions" if res.stage == _lib.STAGE_OPTIONS else ""))
    return workspace if slot is None else buf if res.workspaceSize else None


def grouped_matmul_v4(x: torch.Tensor, weight: torch.Tensor, scale: Optional[torch.Tensor],
                      per_token_scale: Optional[torch.Tensor], group_list: torch.Tensor, *,
                      bias: Optional[torch.Tensor] = None, split_item: int = 3, group_type: int = 0,
                      group_list_type: int = 0, act_type: int = 0, out: Optional[torch.Tensor] = None,
                      out_dtype: torch.dtype = torch.bfloat16, stream=None, workspace: Optional[torch.Tensor] = None,
                      return_workspace: bool = False, out_row_index: Optional[torch.Tensor] = None,
                      out_peers: Optional[Sequence[int]] = None, weight_format: int = ACL_FORMAT_ND,
                      api: str = "V4", tuning_config: Optional[Sequence[int]] = None, quant_group_size: int = 0,
                      options: Optional[LaunchOptions] = None, out_rows: int = 0):
    """y = bf16(act((x @ weight[e]) * scale[e] * per_token_scale)) per expert row range (W8A8), a float16 result with
    ``out_dtype`` torch.float16, or the raw int32 accumulators with torch.int32.  Rows not covered by ``group_list``
    keep their contents.  ``weight_format`` ACL_FORMAT_FRACTAL_NZ: ``weight`` is the 5-D storage of ``format_cast_nz``.
    ``api`` picks the entry point: "V4", "V5" (adds ``tuning_config``) or "WeightNz" (adds ``quant_group_size`` and
    treats the weight as FRACTAL_NZ) - aclnn_grouped_matmul_v5.h:49-58, aclnn_grouped_matmul_weight_nz.h:50-59 of the
    reference.  ``out_row_index`` (int64 [M], an extension of this library) scatters result row r to row
    out_row_index[r]; it goes through the flat entry point gmmB200GroupedMatmulW8A8.  ``options``: per-call
    ``LaunchOptions`` (CTA cap, timing events)."""
    nz = weight_format == ACL_FORMAT_FRACTAL_NZ or api == "WeightNz"
    if out is None and not out_peers:
        n_out = weight.shape[1] * 32 if (nz and weight.dim() == 5) else weight.shape[2]
        out = x.new_empty((x.shape[0], n_out), dtype=out_dtype)
    if out_row_index is not None:
        return _grouped_matmul_flat(x, weight, scale, per_token_scale, group_list, bias, group_list_type, act_type, out,
                                    out_row_index, stream, workspace, return_workspace, out_peers, nz, options, out_rows)
    if api not in _lib.OP_GMM:
        raise ValueError(f"unknown api {api!r}")
    words = _lib.describe_call("tftttttiiiiil", x, (weight, ACL_FORMAT_FRACTAL_NZ if nz else ACL_FORMAT_ND, None), bias, scale, per_token_scale,
                               group_list, out, split_item, group_type, group_list_type, act_type, quant_group_size, _ints(tuning_config))
    workspace = _call(_lib.OP_GMM[api], "aclnnGroupedMatmul" + api, words, x.device, workspace, stream, options)
    return (out, workspace) if return_workspace else out


def _grouped_matmul_flat(x, weight, scale, per_token_scale, group_list, bias, group_list_type, act_type, out, out_row_index,
                         stream, workspace, return_workspace, out_peers=None, nz=False, options=None, out_rows=0):
    """Flat entry point.  ``out_peers`` (device addresses, one [rows, N] bf16 buffer per GPU) makes out_row_index hold
    (gpu << 40) | row; ``out`` may then be None.  ``out_rows``: rows of ``out`` / of every peer buffer (0 = taken from
    ``out``, unbounded without it); rows scattered outside are skipped and reported by ``check_status``."""
    L = _lib.lib()
    M, K = x.shape
    if nz and weight.dim() == 5:
        E, N = weight.shape[0], weight.shape[1] * 32
    else:
        E, _, N = weight.shape
    trans = 2 if nz else int((not weight.is_contiguous()) and weight.transpose(1, 2).is_contiguous())
    for t in (x, scale, per_token_scale, group_list, bias, out, out_row_index):
        if t is not None and not t.is_contiguous():
            raise ValueError("the flat entry point needs contiguous tensors")
    if out_row_index.dtype != torch.int64 or out_row_index.numel() != M:
        raise ValueError("out_row_index must be int64 [M]")
    ydt = _DTYPES[out.dtype] if out is not None else ACL_BF16
    if not out_rows and out is not None:
        out_rows = out.shape[0]
    n_peers = len(out_peers) if out_peers else 0
    peers = (C.c_void_p * max(n_peers, 1))(*[C.c_void_p(a) for a in (out_peers or [])])
    size = C.c_uint64(0)
    rc = L.gmmB200GroupedMatmulW8A8WorkspaceSize(M, K, N, E, ydt, C.byref(size))
    if rc != ACLNN_SUCCESS:
        raise AclnnError(rc, "gmmB200GroupedMatmulW8A8WorkspaceSize")
    p = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731
    handle = _gpu_stream_handle(stream) if x.device.type == "cuda" else _stream_handle(stream)

    def enqueue(workspace):
        rc = L.gmmB200GroupedMatmulW8A8(p(x), p(weight), p(scale), _DTYPES[scale.dtype] if scale is not None else 0, p(per_token_scale),
                                        p(bias), _DTYPES[bias.dtype] if bias is not None else 0, p(group_list), group_list.numel(),
                                        group_list_type, M, K, N, E, trans, act_type, p(out_row_index), peers if n_peers else None, n_peers, out_rows,
                                        p(out), ydt, p(workspace), workspace.numel(), handle,
                                        C.byref(options) if options is not None else None)
        if rc != ACLNN_SUCCESS:
            raise AclnnError(rc, "gmmB200GroupedMatmulW8A8")
    if workspace is None:
        workspace = _with_pooled(x.device, stream, handle, size.value, enqueue)
    else:
        enqueue(workspace)
    return (out, workspace) if return_workspace else out


def grouped_matmul_swiglu_quant(x: torch.Tensor, weight: torch.Tensor, weight_scale: torch.Tensor, x_scale: torch.Tensor,
                                group_list: torch.Tensor, *, bias: Optional[torch.Tensor] = None,
                                offset: Optional[torch.Tensor] = None, output: Optional[torch.Tensor] = None,
                                output_scale: Optional[torch.Tensor] = None, stream=None,
                                workspace: Optional[torch.Tensor] = None, return_workspace: bool = False,
                                weight_format: int = ACL_FORMAT_ND, api: str = "", options: Optional[LaunchOptions] = None):
    """(output int8 [M, N/2], output_scale fp32 [M]) = per-token int8 requant of SwiGLU of the dequantised grouped
    GEMM.  ``group_list`` holds running totals.  Rows at and beyond group_list[-1] keep their contents.
    ``weight_format`` ACL_FORMAT_FRACTAL_NZ: ``weight`` is the 5-D storage of ``format_cast_nz``; ``api`` "WeightNZ"
    calls aclnnGroupedMatmulSwigluQuantWeightNZ (aclnn_grouped_matmul_swiglu_quant_weight_nz.h:37-54 of the reference),
    which takes the storage as FRACTAL_NZ whatever the format says."""
    M = x.shape[0]
    N = weight_scale.shape[1] if weight_scale.dim() == 2 else 0
    if output is None:
        output = x.new_empty((M, N // 2), dtype=torch.int8)
    if output_scale is None:
        output_scale = x.new_empty((M,), dtype=torch.float32)
    words = _lib.describe_call("tfttttttt", x, (weight, weight_format, None), bias, offset, weight_scale, x_scale, group_list, output, output_scale)
    workspace = _call(_lib.OP_SWIGLU_QUANT[api], "aclnnGroupedMatmulSwigluQuant" + api, words, x.device, workspace, stream, options)
    return (output, output_scale, workspace) if return_workspace else (output, output_scale)


def grouped_matmul_finalize_routing(x: torch.Tensor, weight_nz: torch.Tensor, scale: torch.Tensor, group_list: torch.Tensor,
                                    row_index: torch.Tensor, batch: int, *, bias: Optional[torch.Tensor] = None,
                                    pertoken_scale: Optional[torch.Tensor] = None, shared_input: Optional[torch.Tensor] = None,
                                    logit: Optional[torch.Tensor] = None, shared_input_weight: float = 1.0,
                                    shared_input_offset: int = 0, group_list_type: int = 1, out: Optional[torch.Tensor] = None,
                                    view_3d: bool = True, api: str = "", tuning_config: Optional[Sequence[int]] = None,
                                    stream=None, workspace: Optional[torch.Tensor] = None, return_workspace: bool = False,
                                    options: Optional[LaunchOptions] = None):
    """aclnnGroupedMatmulFinalizeRoutingWeightNz (``api`` "") or ...WeightNzV2 (``api`` "V2"): W8A8 grouped GEMM whose fp32
    result rows, weighted by ``logit``, are added into row ``row_index[i]`` of ``out`` [batch, N] on top of the weighted
    ``shared_input`` rows (gmm/grouped_matmul_finalize_routing/op_host/op_api/aclnn_grouped_matmul_finalize_routing_weight_nz.h:48-64
    of the reference).  ``weight_nz`` is the FRACTAL_NZ storage [E, N/32, K/16, 16, 32] (``format_cast_nz``); with
    ``view_3d`` it is described to the operator as the reference's callers do, a view [E, K, N] over that storage."""
    E, n1, k1 = weight_nz.shape[0], weight_nz.shape[1], weight_nz.shape[2]
    N, K = n1 * 32, k1 * 16
    if out is None:
        out = x.new_empty((batch, N), dtype=torch.float32)
    words = _lib.describe_call("tfttttttttiiil", x, (weight_nz, ACL_FORMAT_FRACTAL_NZ, [E, K, N] if view_3d else None), scale, bias,
                               pertoken_scale, group_list, shared_input, logit, row_index, out,
                               struct.unpack("<I", bytes(C.c_float(shared_input_weight)))[0], shared_input_offset, group_list_type, _ints(tuning_config))
    workspace = _call(_lib.OP_FINALIZE_ROUTING[api], "aclnnGroupedMatmulFinalizeRoutingWeightNz" + api, words, x.device, workspace, stream,
                      options)
    return (out, workspace) if return_workspace else out


def grouped_matmul_finalize_routing_flat(x, weight, weight_layout, scale, group_list, row_index, out, *, bias=None,
                                         pertoken_scale=None, shared_input=None, logit=None, shared_input_weight=1.0,
                                         shared_input_offset=0, group_list_type=1, stream=None, workspace=None, options=None):
    """gmmB200GroupedMatmulFinalizeRouting: the same operator without handles; ``weight_layout`` 0 takes the ND [E, K, N]
    weight (the faster layout here), 2 the FRACTAL_NZ storage."""
    L = _lib.lib()
    M, K = x.shape
    if weight_layout == 2:
        E, N = weight.shape[0], weight.shape[1] * 32
    else:
        E, _, N = weight.shape
    p = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731
    handle = _gpu_stream_handle(stream) if x.device.type == "cuda" else _stream_handle(stream)

    def enqueue(workspace):
        rc = L.gmmB200GroupedMatmulFinalizeRouting(
            p(x), p(weight), weight_layout, p(scale), _DTYPES[scale.dtype], p(bias), p(pertoken_scale), p(group_list),
            group_list.numel(), group_list_type, p(shared_input), 0 if shared_input is None else shared_input.shape[0],
            shared_input_offset, shared_input_weight, p(logit), p(row_index), _DTYPES[row_index.dtype], M, K, N, E, p(out),
            out.shape[0], p(workspace), workspace.numel(), handle,
            C.byref(options) if options is not None else None)
        if rc != ACLNN_SUCCESS:
            raise AclnnError(rc, "gmmB200GroupedMatmulFinalizeRouting")
    if workspace is None:
        _with_pooled(x.device, stream, handle, 256, enqueue)
    else:
        enqueue(workspace)
    return out


def moe_init_routing_v3(x: torch.Tensor, expert_idx: torch.Tensor, *, expert_num: int, active_expert_range: Sequence[int],
                        quant_mode: int = 1, scale: Optional[torch.Tensor] = None, offset: Optional[torch.Tensor] = None,
                        active_num: Optional[int] = None, expert_capacity: int = 0, drop_pad_mode: int = 0,
                        expert_tokens_num_type: int = 1, expert_tokens_num_flag: bool = True, row_idx_type: int = 1,
                        outputs=None, stream=None, workspace: Optional[torch.Tensor] = None):
    """aclnnMoeInitRoutingV3 (moe/moe_init_routing_v3/op_host/op_api/aclnn_moe_init_routing_v3.h:24-47 of the reference):
    returns (expandedX, expandedRowIdx, expertTokensCountOrCumsum, expandedScale).  With ``quant_mode`` 1 expandedX is int8
    and expandedScale the per-row scale, i.e. the x / per-token scale of the grouped GEMM operators."""
    n, h = x.shape
    k = expert_idx.shape[1]
    start, end = active_expert_range
    if outputs is None:
        ex = x.new_empty((n * k, h), dtype=torch.int8 if quant_mode == 1 else x.dtype)
        ri = x.new_empty((n * k,), dtype=torch.int32)
        cnt = x.new_empty((end - start,) if expert_tokens_num_type == 1 else (expert_num, 2), dtype=torch.int64)
        es = x.new_empty((n * k,), dtype=torch.float32)
    else:
        ex, ri, cnt, es = outputs
    words = _lib.describe_call("ttttttttiiiiiiiil", x, expert_idx, scale, offset, ex, ri, cnt, es, n * k if active_num is None else active_num,
                               expert_capacity, expert_num, drop_pad_mode, expert_tokens_num_type, 1 if expert_tokens_num_flag else 0, quant_mode,
                               row_idx_type, _ints(active_expert_range))
    _call(_lib.OP_MOE_INIT_ROUTING, "aclnnMoeInitRoutingV3", words, x.device, workspace, stream, None)
    return ex, ri, cnt, es
