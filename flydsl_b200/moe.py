"""Two-stage block-scale MoE layer assembled from the reference-shaped launchers.

The reference ships the two stage kernels and leaves the chaining to its test
(tests/kernels/test_moe_blockscale.py:293-380): routing sort -> stage 1 -> 1x128 re-quantisation ->
stage 2 (-> top-k reduce). ``BlockscaleMoE`` is that chain with persistent buffers, so a step
launches kernels only (sort, gemm1, quant, gemm2[, reduce]) and allocates only the routing arrays after
warm-up, and the result unless ``out`` is given (small blocks: see ``BlockscaleMoE._buffers``).
"""
from __future__ import annotations

from typing import Optional

import torch

from . import _lib
from .kernels.moe_blockscale_2stage import (
    compile_moe_blockscale_gemm1,
    compile_moe_blockscale_gemm2,
    compile_moe_reduction,
)
from .utils import moe_gather_rows, moe_sorting, quant_1x128, quant_pertoken, shuffle_weight

# Scratch that one layer keeps for blocks of at most 32 rows, over all token counts (see _buffers).
_KEPT_SMALL_BYTES = 256 << 20

_DT_NAME = {torch.float16: "f16", torch.bfloat16: "bf16", torch.float32: "f32"}


def _as_torch_stream(stream):
    """torch.cuda.Stream | raw handle | None -> a torch stream object."""
    if stream is None:
        return torch.cuda.current_stream()
    if isinstance(stream, int):
        return torch.cuda.ExternalStream(stream)
    return stream


class BlockscaleMoE:
    """Expert weights (already repacked) plus the launchers and scratch buffers for one layer.

    w1 fp8 ``[E, 2*I, H]`` repacked (gate rows then up rows), w1_scale f32 ``[E, (2I/128)*(H/128)]``;
    w2 fp8 ``[E, H, I]`` repacked, w2_scale f32 ``[E, (H/128)*(I/128)]``.
    ``mode``: "reduce" (per-route store + fixed-order reduce, deterministic) or "atomic".
    """

    def __init__(self, w1, w1_scale, w2, w2_scale, *, topk: int, tile_m: int = 128,
                 mid_dtype=torch.float16, out_dtype=torch.bfloat16, mode: str = "reduce",
                 block_n1: Optional[int] = None, block_n2: Optional[int] = None,
                 sorted_layout: Optional[bool] = None, fused_quant: Optional[bool] = None):
        if mode not in ("reduce", "atomic"):
            raise ValueError(f"mode must be 'reduce' or 'atomic', got {mode!r}")
        self.E, two_i, self.H = w1.shape
        self.I = two_i // 2
        if tuple(w2.shape) != (self.E, self.H, self.I):
            raise ValueError(f"w2 shape {tuple(w2.shape)} does not match w1 {tuple(w1.shape)}")
        self.w1, self.w2 = w1, w2
        self.w1_scale = w1_scale.contiguous().view(-1)
        self.w2_scale = w2_scale.contiguous().view(-1)
        self.topk, self.tile_m, self.mode = int(topk), int(tile_m), mode
        self.mid_dtype, self.out_dtype = mid_dtype, out_dtype
        # Routing-order intermediates: activations are permuted once (one bandwidth-bound pass) and
        # both stages then fetch their A tiles with TMA instead of gathering rows with cp.async;
        # the stage-1 output and its re-quantisation stay in routing order as well.
        # Measured on the 256-expert layer: 4.31 -> 3.76 ms at 128-token blocks, but slightly slower
        # for decode-size batches (one more launch, nothing to hide), hence the default by block size.
        # Blocks of at most 32 rows take these layouts all the same where forward() does the routing
        # itself and it pays off (_small_pays_off): the stages are then the kernel with the weights on the
        # MMA's M side.
        self.sorted_layout = (self.tile_m >= 64 and self.tile_m % 8 == 0) if sorted_layout is None \
            else bool(sorted_layout)
        # Optional: re-quantisation between the stages fused into the stage-1 epilogue (routing-order
        # layouts, 256-wide stage-1 tiles): the 16-bit intermediate is never written. Bit-identical,
        # but measured 3 % slower on the 256-expert layer (the heavier tile epilogue stalls the MMA
        # pipe longer than the separate quantiser kernel takes), so it is off unless asked for.
        can_fuse = self.sorted_layout and block_n1 in (None, 0, 256)
        self.fused_quant = False if fused_quant is None else bool(fused_quant)
        if self.fused_quant and not can_fuse:
            raise ValueError("fused_quant needs sorted_layout and block_n1 in (None, 256)")
        common = dict(model_dim=self.H, inter_dim=self.I, experts=self.E, topk=self.topk,
                      tile_m=self.tile_m, tile_n=256, tile_k=128)

        def stages(in_order):
            return (compile_moe_blockscale_gemm1(doweight_stage1=False, out_dtype=_DT_NAME[mid_dtype],
                                                 block_n=block_n1, a_sorted=in_order, out_sorted=in_order, **common),
                    compile_moe_blockscale_gemm2(doweight_stage2=True, out_dtype=_DT_NAME[out_dtype],
                                                 accumulate=(mode == "atomic"), block_n=block_n2, a_sorted=in_order,
                                                 **common))

        self.gemm1, self.gemm2 = stages(self.sorted_layout)
        small = sorted_layout is None and self.tile_m <= 32 and self.tile_m % 8 == 0 and not (block_n1 or block_n2)
        self._small_stages = stages(True) if small else None
        self.reduce = compile_moe_reduction(topk=self.topk, model_dim=self.H,
                                            dtype_str=_DT_NAME[out_dtype]) if mode == "reduce" else None
        self._buf = {}
        self._kept_small = 0

    @classmethod
    def from_unpacked(cls, w1_q, w1_scale, w2_q, w2_scale, **kw):
        """Build from plain row-major fp8 weights (repacks them on the GPU)."""
        return cls(shuffle_weight(w1_q), w1_scale, shuffle_weight(w2_q), w2_scale, **kw)

    def _buffers(self, T: int, dev, in_order: Optional[bool] = None):
        """Scratch for T tokens, kept by token count. The routing-order buffers of small blocks are mostly
        padding (256 experts of 7168 x 2048: 63 MB for 32 tokens in blocks of 16, 170 MB for 256 in blocks of
        32), and a server meets every batch size: they are kept up to _KEPT_SMALL_BYTES per layer, and beyond
        that a call takes its own from torch's allocator (about 10 us on the host) and gives them back. Nothing
        kept is ever freed or shared between token counts, so captured graphs and calls on other streams
        find it as they left it."""
        in_order = self.sorted_layout if in_order is None else in_order
        key = (T, dev, in_order)
        b = self._buf.get(key)
        if b is None:
            # rows of padding positions are never written and never looked at, whatever they hold; the
            # layouts that a caller's routing can meet start out as zeros all the same
            small = in_order and not self.sorted_layout
            new = torch.empty if small else torch.zeros
            # rows of the stage-1 output / stage-2 input: routes, or sorted positions incl. padding
            L = (T * self.topk + self.E * self.tile_m - self.topk) if in_order else T * self.topk
            b = {
                "rows": L,
                "x_sorted": torch.empty((L, self.H), dtype=torch.float8_e4m3fn, device=dev)
                if in_order else None,
                "xs_sorted": torch.empty((self.H // 128, L), dtype=torch.float32, device=dev)
                if in_order else None,
                "out1": None if self.fused_quant else new((L, self.I), dtype=self.mid_dtype, device=dev),
                "a2_q": new((L, self.I), dtype=torch.uint8, device=dev).view(torch.float8_e4m3fn),
                "a2_s": new((self.I // 128, L), dtype=torch.float32, device=dev),
                "routes": torch.empty((T * self.topk, self.H), dtype=self.out_dtype, device=dev)
                if self.mode == "reduce" else None,
            }
            if small:
                nbytes = sum(t.numel() * t.element_size() for t in b.values() if torch.is_tensor(t))
                if self._kept_small + nbytes > _KEPT_SMALL_BYTES:
                    return b
                self._kept_small += nbytes
            self._buf[key] = b
        return b

    def _small_pays_off(self, T: int) -> bool:
        """Whether T tokens in blocks of at most 32 rows take routing-order layouts. The stages gain from
        blocks that follow one another in the same expert (one pass over its weights for two) and, in a
        steady stream of calls, from the tensor work that is not done for padding; the permute costs 5 to 20 us.
        Measured in steady streams, routing order / gathered (us a layer; uniform routing, and with every 16th expert
        hot):
          blocks of 16  256 experts of 7168 x 2048, top 8, 12 tokens 582 / 708 and 331 / 349, 32 tokens 1087 / 1330 and 543 /
                        605, 128 x 4096 x 1536, 64 tokens 389 / 424 and 357 / 427, 8 tokens 187 / 187 and 141 / 131, 256 x
                        3072 x 1024, top 4, 128 tokens 343 / 370 and 158 / 164, 32 tokens 184 / 185 and 93 / 84, 64 x 2048 x
                        1024, top 6, 200 tokens 116 / 133 and 128 / 134, 128 tokens 109 / 100 and 107 / 115, 64 tokens 124 /
                        100 and 101 / 99
          blocks of 32  256 x 7168 x 2048, 64 tokens 1522 / 1818 and 871 / 1014, 256 tokens 1744 / 2078 and 1725 / 2177, 128 x
                        4096 x 1536, 256 tokens 440 / 454 and 469 / 547, 128 tokens 428 / 442 and 429 / 483, 512 tokens 486 /
                        683 and 532 / 664, 256 x 3072 x 1024, 384 tokens 441 / 455 and 317 / 341, 64 x 2048 x 1024, 256 tokens
                        123 / 104 and 123 / 120, 384 tokens 129 / 142 and 145 / 141
        Over 120 drawn layers the choice is 0.7 % slower than the faster side on average (two of them by more than
        10 %). Graph replays of the same layers leave the clock higher and move the crossings up: there blocks of 32 with
        less than a tenth of a block per expert are up to 15 % faster gathered;
        and with more blocks than the kernel lists: see moe_swap_pays_off in blockscale_gemm.cu."""
        routes, rows = T * self.topk, self.E * self.tile_m
        if self.tile_m > 16 and routes + rows - self.topk > 4096 * self.tile_m:
            return False
        nbytes = min(self.E, routes) * 3 * self.H * self.I   # weights of the experts that may be hit
        if nbytes >= 4e9:
            return True
        least = 0.75 if nbytes < 1e9 else 0.1 if self.tile_m <= 16 else 0.5
        return routes >= least * rows

    def forward(self, x_q, x_scale_t, topk_ids, topk_weights, out=None, stream=None,
                routing=None):
        """x_q fp8 ``[T, H]``; x_scale_t f32 ``[H/128, T]``; topk_ids i32 ``[T, k]``; topk_weights f32.
        Returns ``out [T, H]``. ``routing`` may carry precomputed sort buffers
        ``(sorted_ids, sorted_weights, sorted_expert_ids, num_valid_ids)``."""
        if stream is None:   # the current stream: every launch below takes it by itself
            return self._forward(x_q, x_scale_t, topk_ids, topk_weights, out, routing)
        with torch.cuda.stream(_as_torch_stream(stream)):
            return self._forward(x_q, x_scale_t, topk_ids, topk_weights, out, routing)

    def _forward(self, x_q, x_scale_t, topk_ids, topk_weights, out, routing):
        # every launch below goes to torch's current stream (stream=None)
        T = x_q.shape[0]
        dev = x_q.device
        dense_in = x_q.is_contiguous() and x_scale_t.is_contiguous()
        small = (self._small_stages is not None and routing is None and dense_in
                 and topk_ids.shape == (T, self.topk)   # the fused permute takes no other routing
                 and self._small_pays_off(T))
        gemm1, gemm2 = self._small_stages if small else (self.gemm1, self.gemm2)
        in_order = self.sorted_layout or small
        b = self._buffers(T, dev, in_order)
        permuted = False
        if routing is None:
            # routing-order layouts: the sort kernel also permutes the activations (one launch)
            fuse = in_order and dense_in
            sid, sw, seid, npp = moe_sorting(
                topk_ids, topk_weights, num_experts=self.E, block_size=self.tile_m,
                permute=(x_q, x_scale_t, b["x_sorted"], b["xs_sorted"]) if fuse else None)
            permuted = fuse
        else:
            sid, sw, seid, npp = routing
        nblk = seid.numel()
        mid_code = {torch.float16: _lib.F16, torch.bfloat16: _lib.BF16}[self.mid_dtype]
        if in_order:
            if sid.numel() != b["rows"]:
                raise ValueError("routing buffers do not match this layer's experts/tile_m/topk")
            if not permuted:
                moe_gather_rows(x_q, x_scale_t, sid, npp, topk=self.topk, out=b["x_sorted"],
                                scale_out=b["xs_sorted"])
            if self.fused_quant:
                gemm1.quantized(b["a2_q"], b["a2_s"], b["x_sorted"], self.w1, b["xs_sorted"],
                                self.w1_scale, sid, seid, sw, npp, T, nblk, None)
            else:
                gemm1(b["out1"], b["x_sorted"], self.w1, b["xs_sorted"], self.w1_scale, sid, seid, sw,
                      npp, T, self.I, self.H, nblk, None)
                _lib.check(_lib.load().flyb200_quant_1x128_routes(
                    b["out1"].data_ptr(), b["a2_q"].data_ptr(), b["a2_s"].data_ptr(), npp.data_ptr(),
                    sid.data_ptr(), T, self.topk, b["rows"], self.I, mid_code, _lib.stream_handle(None)))
        else:
            gemm1(b["out1"], x_q, self.w1, x_scale_t, self.w1_scale, sid, seid, sw, npp, T, self.I,
                  self.H, nblk, None)
            _lib.check(_lib.load().flyb200_quant_1x128(
                b["out1"].data_ptr(), b["a2_q"].data_ptr(), b["a2_s"].data_ptr(), T * self.topk, self.I,
                mid_code, _lib.stream_handle(None)))
        if out is None:
            out = torch.empty((T, self.H), dtype=self.out_dtype, device=dev)
        if self.mode == "atomic":
            out.zero_()
            gemm2(out, b["a2_q"], self.w2, b["a2_s"], self.w2_scale, sid, seid, sw, npp, T,
                  self.H, self.I, nblk, None)
        else:
            if routing is not None:
                # A caller's routing may drop routes (expert_mask, ids outside the local experts):
                # their rows are never written by stage 2, so they must read as zero in the sum
                # (the reference wrapper zero-fills its intermediate, :2714-2715).
                b["routes"].zero_()
            gemm2(b["routes"], b["a2_q"], self.w2, b["a2_s"], self.w2_scale, sid, seid, sw, npp,
                  T, self.H, self.I, nblk, None)
            self.reduce(b["routes"], out, None, T, None)
        return out

    #: kernels one forward() launches (sort[+permute], gemm1, quant, gemm2, reduce | memset+gemm2)
    @property
    def launches_per_step(self) -> int:
        return 4 if (self.sorted_layout and self.fused_quant) else 5



class PertokenMoE:
    """The same chain for the per-token-scale sibling (kernels/moe_gemm_2stage.py of the reference,
    fp8): routing sort -> permute into routing order -> stage 1 -> whole-row re-quantisation -> stage
    2 -> top-k reduce, with persistent buffers. The reference test chains the stage kernels by hand
    and re-quantises with torch on the host side (tests/kernels/test_moe_gemm.py:1236-1330); here
    every step is a kernel of this library.

    w1 fp8 ``[E, 2*I, H]`` repacked (gate rows then up rows), w1_scale f32 ``[E*2*I]`` (one per output
    channel); w2 fp8 ``[E, H, I]`` repacked, w2_scale f32 ``[E*H]``. Activations come with one scale
    per token. ``tile_m`` must be a multiple of 8 (routing-order layouts are always used).
    """

    def __init__(self, w1, w1_scale, w2, w2_scale, *, topk: int, tile_m: int = 128,
                 mid_dtype=torch.float16, out_dtype=torch.bfloat16):
        from .kernels.moe_gemm_2stage import compile_moe_gemm1, compile_moe_gemm2

        self.E, two_i, self.H = w1.shape
        self.I = two_i // 2
        if tuple(w2.shape) != (self.E, self.H, self.I):
            raise ValueError(f"w2 shape {tuple(w2.shape)} does not match w1 {tuple(w1.shape)}")
        if int(tile_m) % 8:
            raise ValueError(f"tile_m must be a multiple of 8, got {tile_m}")
        self.w1, self.w2 = w1, w2
        self.w1_scale = w1_scale.contiguous().view(-1)
        self.w2_scale = w2_scale.contiguous().view(-1)
        self.topk, self.tile_m = int(topk), int(tile_m)
        self.mid_dtype, self.out_dtype = mid_dtype, out_dtype
        common = dict(model_dim=self.H, inter_dim=self.I, experts=self.E, topk=self.topk,
                      tile_m=self.tile_m, tile_n=256, tile_k=128, in_dtype="fp8")
        self.gemm1 = compile_moe_gemm1(doweight_stage1=False, out_dtype=_DT_NAME[mid_dtype], a_sorted=True,
                                       out_sorted=True, **common)
        self.gemm2 = compile_moe_gemm2(doweight_stage2=True, out_dtype=_DT_NAME[out_dtype], accumulate=False,
                                       a_sorted=True, **common)
        self.reduce = compile_moe_reduction(topk=self.topk, model_dim=self.H, dtype_str=_DT_NAME[out_dtype])
        self._buf = {}

    @classmethod
    def from_unpacked(cls, w1_q, w1_scale, w2_q, w2_scale, **kw):
        """Build from plain row-major fp8 weights (repacks them on the GPU)."""
        return cls(shuffle_weight(w1_q), w1_scale, shuffle_weight(w2_q), w2_scale, **kw)

    def _buffers(self, T: int, dev):
        key = (T, dev)
        b = self._buf.get(key)
        if b is None:
            L = T * self.topk + self.E * self.tile_m - self.topk   # sorted positions incl. padding
            b = {
                "rows": L,
                "x_sorted": torch.empty((L, self.H), dtype=torch.float8_e4m3fn, device=dev),
                "xs_sorted": torch.ones((L,), dtype=torch.float32, device=dev),
                "out1": torch.zeros((L, self.I), dtype=self.mid_dtype, device=dev),
                "a2_q": torch.zeros((L, self.I), dtype=torch.uint8, device=dev).view(torch.float8_e4m3fn),
                "a2_s": torch.ones((L,), dtype=torch.float32, device=dev),
                "routes": torch.empty((T * self.topk, self.H), dtype=self.out_dtype, device=dev),
            }
            self._buf[key] = b
        return b

    def forward(self, x_q, x_scale, topk_ids, topk_weights, out=None, stream=None, routing=None):
        """x_q fp8 ``[T, H]``; x_scale f32 ``[T]`` (or ``[T, 1]``); topk_ids i32 ``[T, k]``; topk_weights
        f32. Returns ``out [T, H]``. ``routing`` may carry precomputed sort buffers
        ``(sorted_ids, sorted_weights, sorted_expert_ids, num_valid_ids)``."""
        if stream is None:   # the current stream: every launch below takes it by itself
            return self._forward(x_q, x_scale, topk_ids, topk_weights, out, routing)
        with torch.cuda.stream(_as_torch_stream(stream)):
            return self._forward(x_q, x_scale, topk_ids, topk_weights, out, routing)

    def _forward(self, x_q, x_scale, topk_ids, topk_weights, out, routing):
        T = x_q.shape[0]
        dev = x_q.device
        b = self._buffers(T, dev)
        if routing is None:
            sid, sw, seid, npp = moe_sorting(topk_ids, topk_weights, num_experts=self.E,
                                             block_size=self.tile_m)
        else:
            sid, sw, seid, npp = routing
        if sid.numel() != b["rows"]:
            raise ValueError("routing buffers do not match this layer's experts/tile_m/topk")
        nblk = seid.numel()
        moe_gather_rows(x_q, x_scale.reshape(-1), sid, npp, topk=self.topk, out=b["x_sorted"],
                        scale_out=b["xs_sorted"], per_token=True)
        self.gemm1(b["out1"], b["x_sorted"], self.w1, b["xs_sorted"], self.w1_scale, sid, seid, sw, npp,
                   T, self.I, self.H, nblk, None)
        quant_pertoken(b["out1"], npp, out=b["a2_q"], scale_out=b["a2_s"])
        if out is None:
            out = torch.empty((T, self.H), dtype=self.out_dtype, device=dev)
        if routing is not None:
            b["routes"].zero_()   # a caller's routing may drop routes: their rows must sum as zero
        self.gemm2(b["routes"], b["a2_q"], self.w2, b["a2_s"], self.w2_scale, sid, seid, sw, npp, T,
                   self.H, self.I, nblk, None)
        self.reduce(b["routes"], out, None, T, None)
        return out

    #: kernels one forward() launches: sort, permute, gemm1, quant, gemm2, reduce
    launches_per_step = 6
