"""What parts share at run time: device, run dtype, the status word, and the matrix product.

``Runtime.linear`` is the one place where ``y = x W^T`` is computed.  The reference computes its
unquantised linears with a library call (``F.linear``, pygguf_engine/quant_kernels.py:1836); here
the library product (cuBLAS through ``torch.mm``) stands wherever the package's own tensor-core
kernels do not take the shape, and the float32 mode never computes in less than float32 (TF32 is
switched off around the call; larger products of 16 rows and more split each operand into three
bfloat16 parts, csrc/gemm_split32.cu).
"""
from __future__ import annotations

import os
from typing import Dict, Optional, Tuple

import torch

from ..kernels import KernelError, ops

STATUS_MESSAGES = {
    1: "a token id is outside the embedding table (token row {0}, id {1}, vocabulary {2})",
    2: "a cache page number is outside the pool ({0}, page {1}, {2})",
    3: "a position is beyond the position tables or the page table (token {0}, position {1}, limit {2})",
    4: "a bounded wait inside a kernel ran out (where {0}, detail {1}, {2})",
    5: "a slot number is outside the cache ({0}, {1}, {2})",
}


def _reductions_switch() -> tuple:
    """How ``torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction`` is read and set: as (allowed, split-K allowed) and
    without its parsing where this PyTorch has the calls behind it (every library product asks, and a prompt's step has three of
    them a layer), else as the attribute itself."""
    read = getattr(torch._C, "_get_cublas_allow_bf16_reduced_precision_reduction", None)
    write = getattr(torch._C, "_set_cublas_allow_bf16_reduced_precision_reduction", None)
    if read is not None and write is not None and isinstance(read(), tuple) and len(read()) == 2:
        return read, write
    matmul = torch.backends.cuda.matmul
    return (lambda: (matmul.allow_bf16_reduced_precision_reduction, True),
            lambda allowed, split_k: setattr(matmul, "allow_bf16_reduced_precision_reduction", allowed))


_reduced_reductions, _set_reduced_reductions = _reductions_switch()


class PendingTokens:
    """Tokens (and the status word) on their way to the host; ``result()`` waits and returns the tokens,
    raising if a kernel reported an error."""

    def __init__(self, runtime: "Runtime") -> None:
        self.runtime = runtime
        self.host = torch.empty(4 + runtime.max_result_rows, dtype=torch.int32, pin_memory=runtime.is_cuda)
        self.event = torch.cuda.Event() if runtime.is_cuda else None
        self.n = 0

    def start(self, n: int) -> None:
        self.n = n
        self.host[:4 + n].copy_(self.runtime._status_and_tokens[:4 + n], non_blocking=True)
        if self.event is not None:
            self.event.record()

    def result(self):
        if self.event is not None:
            self.event.synchronize()
        vals = self.host[:4 + self.n].tolist()
        if vals[0] != 0:
            self.runtime.status.zero_()
            msg = STATUS_MESSAGES.get(vals[0], "kernel status {0}").format(*vals[1:4])
            raise KernelError(f"a kernel reported an error during the step: {msg}")
        return vals[4:]


def large_gemm_fill(rows: int, cols: int, sms: int) -> float:
    """Share of busy tile slots when ``rows x cols`` outputs are cut into 256 x 256 tiles and run in
    waves of one tile per pair of SMs: 96 tiles on 74 pairs need two waves and fill 0.65 of them."""
    tiles = -(-rows // 256) * -(-cols // 256)
    pairs = max(1, sms // 2)
    waves = -(-tiles // pairs)
    return tiles / (waves * pairs)


def split32_pays(rows: int, cols: int, depth: int) -> bool:
    """Whether a float32 product of 16 rows or more is faster on csrc/gemm_split32.cu than in the library.  It has two or three
    launches and a long start, so sums of few terms pay only where the outputs are many; up to 16 rows the library has a
    short-cut for narrow weights.  This kernel and the library, us: 24 rows, 4,096 x 1,024 weights 13 and 27; 16 rows, 151,936 x
    1,024 222 and 238, 256 x 1,024 10.4 and 8.6; 128 rows, 4,096 x 512 12 and 17, 1,024 x 512 11.2 and 10.9; 512 rows, 1,024 x 64 5.8
    and 4.4; 2,048 rows, 4,096 x 64 25 and 35.  Over 1,430 sizes (16 to 4,096 rows, 16 to 32,768 columns, 32 to 1,536 terms) the
    choice is nowhere more than 4 % slower than the library, and misses a gain of 10 % or more in one of 36."""
    if depth < 64:
        return False
    if depth < 768:
        return rows >= 96 and rows * cols >= 3 << (19 if depth < 128 else 18 if depth < 512 else 17)
    return depth >= 1536 or ((rows > 16 or cols >= 2048) and (cols >= 128 or rows <= 1024))


class Runtime:
    def __init__(self, device, dtype: torch.dtype) -> None:
        self.device = torch.device(device)
        if dtype not in (torch.float32, torch.bfloat16):
            raise KernelError(f"run dtype must be float32 or bfloat16, got {dtype}")
        self.dtype = dtype
        self.is_cuda = self.device.type == "cuda"
        # the status word (4 ints) and, right behind it, room for the tokens a sampler draws: one
        # device-to-host copy then brings both
        self.max_result_rows = 8192
        self._status_and_tokens = torch.zeros(4 + self.max_result_rows, dtype=torch.int32, device=self.device)
        self.status = self._status_and_tokens[:4]
        self.token_area = self._status_and_tokens[4:]
        self._host_result = None
        self._pending_ring = None
        self._pending_next = 0
        self._adopted: Dict[Tuple[int, torch.dtype], torch.Tensor] = {}
        self.position_limit = None  # the longest sequence the engine holds: position tables need no more rows
        self.generic_attention = os.environ.get("PE_B200_GENERIC_ATTENTION", "0") == "1"  # comparisons: no tensor-core attention
        self.gemm_backend = None  # a callable (x, weight, out, out_dtype) -> tensor or None that takes over products
        self.own_small_gemm = True  # products with few rows run on csrc/gemm_smallm.cu
        self.small_gemm_rows = 8    # up to this many rows (measured: beyond it the library product is faster)
        self.chain_norms = True     # norms of few rows ride in the products around them (parts/block.py, PreNormBlock): blocks
        self.chain_widths = (512, {8: 1024, 12: 4096, 32: 2048})   # of this width at least and, by the most rows, at most
        # products with many rows run on csrc/gemm_umma.cu (tcgen05 + TMA); in between, and for shapes it
        # refuses, the library product stands (measured: with fewer rows too few tiles exist to fill the SMs)
        self.own_large_gemm = True
        self.large_gemm_rows = 1024
        self.large_gemm_min_fill = 0.8   # least share of the waves of tiles that does work (see takes_large_gemm)
        # float32 products with at least this many rows may run on csrc/gemm_split32.cu (see split32_pays)
        self.split32_rows = 16
        self.pair_gemm = True       # large products on tcgen05 cta_group::2
        # q/k-norm, rotation and cache append in the epilogue of the q|k|v product where the pair kernel runs it
        # (PE_B200_FUSE_QKV_ROPE=0 keeps them kernels of their own, for comparisons)
        self.fuse_qkv_rope = os.environ.get("PE_B200_FUSE_QKV_ROPE", "1") != "0"

    # ---- weights -------------------------------------------------------------------------
    def adopt(self, tensor: torch.Tensor, dtype: Optional[torch.dtype] = None) -> torch.Tensor:
        """The tensor on the run device in ``dtype`` (default: the run dtype), converted once even if
        several parts use it (tied embedding and output head share one copy)."""
        dtype = dtype or self.dtype
        key = (id(tensor), dtype)
        got = self._adopted.get(key)
        if got is None:
            got = tensor.to(device=self.device, dtype=dtype).contiguous()
            self._adopted[key] = got
        return got

    def forget_adopted(self) -> None:
        self._adopted.clear()

    # ---- status word -----------------------------------------------------------------------
    def raise_on_status(self) -> None:
        """Read the kernels' status word (one small device-to-host copy) and raise if it is set."""
        s = self.status.tolist()
        if s[0] != 0:
            self.status.zero_()
            msg = STATUS_MESSAGES.get(s[0], "kernel status {0}").format(*s[1:])
            raise KernelError(f"a kernel reported an error during the step: {msg}")

    def takes_small_gemm(self, x: torch.Tensor, weight: torch.Tensor) -> bool:
        return (self.own_small_gemm and x.dim() == 2 and x.shape[0] <= self.small_gemm_rows
                and ops.gemm_smallm_supported(x, weight))

    def takes_chained(self, rows: int, width: int) -> bool:
        """Whether a step of so many rows of ``width`` may run a pre-norm block as a chain of products (csrc/gemm_smallm.cu, CHAIN).
        A decode step of 28 layers of width 1,024, chained : with norms of their own: 1 row 698 : 727 us, 8 rows 921 : 964, 9 rows
        1,143 : 1,632 (where the library's products begin otherwise), 16 rows 1,281 : 1,750, 24 rows 1,635 : 1,922, 32 rows 1,817 :
        2,090.  Width 2,048: 1 row 463 : 468, 4 rows 649 : 563, 8 rows 765 : 659, 9 rows 779 : 942, 24 rows 1,197 : 1,252, 32 rows 1,373 :
        1,414.  Width 4,096: 1 row 1,409 : 1,252, 12 rows 1,723 : 1,841, 24 rows 2,147 : 2,004.  A row's squares come in a part per 16
        features, which every block adds up again, and each block reads its rows from L2.
        Narrower models keep their norms, which is no rule of speed: a decode step and a prompt of the same tokens then round alike (at
        width 96 the two were 2.4 % of the logits apart after hundreds of chained steps).  In the 2-norm of the logits of three layers a
        chained step is 0.4, 0.6 and 0.9 % off the prompt of the same tokens at widths 512, 1,024 and 2,048, one with norms of its own as
        much, and both 0.5, 0.7 and 1.1 % off float32."""
        return (self.chain_norms and self.is_cuda and self.dtype == torch.bfloat16 and self.own_small_gemm and self.gemm_backend is None
                and self.chain_widths[0] <= width <= next((w for r, w in self.chain_widths[1].items() if rows <= r), 0))

    def takes_large_gemm(self, x: torch.Tensor, weight: torch.Tensor, pair_offset: int = 0) -> bool:
        rows = 9 if pair_offset else self.large_gemm_rows   # the fused gate wins at every size above the small kernel's
        if not (self.own_large_gemm and x.dim() == 2 and x.shape[0] >= rows
                and ops.gemm_umma_supported(x, weight, pair_offset)):
            return False
        # A plain product whose 256 x 256 tiles leave the last wave of SM pairs mostly idle goes to the
        # library, which has smaller tiles to choose from (8B shape, 1,536 rows, down projection: 96 tiles
        # on 74 pairs took 133 us against 103 us).
        return bool(pair_offset) or large_gemm_fill(x.shape[0], weight.shape[0], ops.sm_count(x.device)) >= self.large_gemm_min_fill

    def takes_split32_gemm(self, x: torch.Tensor, weight: torch.Tensor, out: Optional[torch.Tensor], out_dtype) -> bool:
        """Whether a float32 product runs on csrc/gemm_split32.cu (float32's precision on the tensor cores)."""
        return (x.dtype == torch.float32 and self.own_large_gemm and x.dim() == 2 and x.shape[0] >= self.split32_rows
                and out_dtype in (None, torch.float32) and split32_pays(x.shape[0], weight.shape[0], x.shape[1]) and ops.gemm_split32_supported(x, weight)
                and (out is None or (out.dtype == torch.float32 and out.stride(1) == 1 and out.stride(0) % 4 == 0
                                     and out.stride(0) >= weight.shape[0] and out.data_ptr() % 16 == 0))
                and (out is not None or weight.shape[0] % 4 == 0))

    def fetch_tokens(self, n: int):
        """The first ``n`` ints of ``token_area`` as a list, after checking the status word: one
        device-to-host copy for both (the copy waits for the step's kernels)."""
        if self._host_result is None:
            self._host_result = torch.empty(4 + self.max_result_rows, dtype=torch.int32,
                                            pin_memory=self.is_cuda)
        host = self._host_result[:4 + n]
        host.copy_(self._status_and_tokens[:4 + n], non_blocking=True)
        if self.is_cuda:
            torch.cuda.current_stream(self.device).synchronize()
        vals = host.tolist()
        if vals[0] != 0:
            self.status.zero_()
            msg = STATUS_MESSAGES.get(vals[0], "kernel status {0}").format(*vals[1:4])
            raise KernelError(f"a kernel reported an error during the step: {msg}")
        return vals[4:]

    def fetch_tokens_async(self, n: int) -> "PendingTokens":
        """Start the copy of the status word and the first ``n`` ints of ``token_area`` to the host and
        return at once; ``result()`` of the returned handle waits for it.  The device may go on and
        overwrite ``token_area`` meanwhile: the copy is ordered before whatever is launched next."""
        if self._pending_ring is None:
            self._pending_ring = [PendingTokens(self) for _ in range(4)]
            self._pending_next = 0
        h = self._pending_ring[self._pending_next]
        self._pending_next = (self._pending_next + 1) % len(self._pending_ring)
        h.start(n)
        return h

    # ---- matrix products ---------------------------------------------------------------------
    def batched_linear(self, xs: torch.Tensor, weights: torch.Tensor, out: torch.Tensor) -> torch.Tensor:
        """``out[i] = xs[i] @ weights[i]^T`` for ``xs [G, M, K]``, ``weights [G, N, K]``: several projections, each of an
        input of its own, as one library call (float32: true float32; bfloat16: float32 accumulation)."""
        if not self.is_cuda:
            raise KernelError("this package computes on a CUDA device only; there is no CPU path")
        tf32 = torch.backends.cuda.matmul.allow_tf32
        red = torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction
        torch.backends.cuda.matmul.allow_tf32 = False
        torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
        try:
            return torch.bmm(xs, weights.transpose(1, 2), out=out)
        finally:
            torch.backends.cuda.matmul.allow_tf32 = tf32
            torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = red

    def linear(self, x: torch.Tensor, weight: torch.Tensor, out: Optional[torch.Tensor] = None,
               out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
        """``x [M, K] @ weight [N, K]^T -> [M, N]``."""
        if not self.is_cuda:
            raise KernelError("this package computes on a CUDA device only; there is no CPU path")
        if self.gemm_backend is not None:
            y = self.gemm_backend(x, weight, out, out_dtype)
            if y is not None:
                return y
        if self.takes_large_gemm(x, weight):
            if out is None:
                out = torch.empty((x.shape[0], weight.shape[0]), dtype=out_dtype or x.dtype, device=x.device)
            # two SMs per 256 x 256 tile (csrc/gemm_umma2.cu): measured 3-6 % faster than one SM per
            # 128 x 256 tile on the plain products; the fused gate|up product stays on gemm_umma.cu
            pair = self.pair_gemm and ops.gemm_umma2_supported(x, weight)
            (ops.gemm_umma2 if pair else ops.gemm_umma)(x, weight, out, self.status)
            return out
        if self.takes_small_gemm(x, weight):
            # a handful of rows: the package's weight-streaming kernel (csrc/gemm_smallm.cu)
            if out is None:
                out = torch.empty((x.shape[0], weight.shape[0]), dtype=out_dtype or x.dtype, device=x.device)
            ops.gemm_smallm(x, weight, out)
            return out
        if self.takes_split32_gemm(x, weight, out, out_dtype):
            if out is None:
                out = torch.empty((x.shape[0], weight.shape[0]), dtype=torch.float32, device=x.device)
            ops.gemm_split32(x, weight, out, self.status)
            return out
        if x.dtype == torch.float32:
            prev = torch.backends.cuda.matmul.allow_tf32
            if prev:
                torch.backends.cuda.matmul.allow_tf32 = False
            try:
                return torch.mm(x, weight.t(), out=out) if out is not None else torch.mm(x, weight.t())
            finally:
                if prev:
                    torch.backends.cuda.matmul.allow_tf32 = True
        # library product in bfloat16: keep its reductions in float32
        prev = _reduced_reductions()
        if prev[0]:
            _set_reduced_reductions(False, True)
        try:
            if out_dtype is not None and out_dtype != x.dtype:
                y = torch.mm(x, weight.t(), out_dtype=out_dtype)
                if out is not None:
                    out.copy_(y)
                    return out
                return y
            return torch.mm(x, weight.t(), out=out) if out is not None else torch.mm(x, weight.t())
        finally:
            if prev[0]:
                _set_reduced_reductions(*prev)
