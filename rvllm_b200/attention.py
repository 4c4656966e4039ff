"""FP8-KV paged GQA decode attention: host mirror of PagedDecodeParams and
PagedDecodeFp8Launcher (v3/crates/rvllm-attention/src/decode.rs:14-102,458-711)."""
from __future__ import annotations

from dataclasses import dataclass

from . import _lib
from ._lib import BF16, F16, check, lib, native


_f16 = None


def _float16():
    global _f16
    if _f16 is None:
        import torch

        _f16 = torch.float16
    return _f16


@dataclass
class PagedDecodeParams:
    num_seqs: int
    num_heads: int
    num_kv_heads: int
    head_dim: int
    block_size: int
    max_blocks_per_seq: int
    num_blocks_total: int
    scale: float
    window_size_left: int = -1

    def validate(self) -> None:
        check(lib().rvllm_paged_decode_fp8_validate(self.num_seqs, self.num_heads, self.num_kv_heads, self.head_dim,
                                                    self.block_size, self.max_blocks_per_seq, self.num_blocks_total,
                                                    self.window_size_left, self.scale), "PagedDecodeParams.validate")

    def workspace_bytes(self) -> int:
        n = int(lib().rvllm_paged_decode_workspace_size(self.num_seqs, self.num_heads, self.num_kv_heads, self.head_dim))
        if n == 2 ** 64 - 1:
            raise _lib.InvalidArgument(_lib.E_INVALID, "workspace_bytes", "shape rejected by the workspace query")
        return n

    def max_chunks(self) -> int:
        return int(lib().rvllm_paged_decode_max_chunks(self.num_seqs, self.num_kv_heads))


class PagedDecodeFp8Launcher:
    """launch(): q [B, H, HD] u8, caches [blocks, block_size, KVH, HD] u8, out [B, H, HD] 16-bit."""

    def __init__(self, params: PagedDecodeParams):
        self.params = params

    def launch(self, q_fp8, k_cache, v_cache, out, block_tables, context_lens, workspace=None, k_scale_cache=None,
               v_scale_cache=None, q_scale_cache=None, q_descale=None, k_descale=None, v_descale=None,
               stream=None) -> None:
        p = self.params
        rc = native().rvllm_paged_decode_fp8(q_fp8, k_cache, v_cache, out, F16 if out.dtype == _float16() else BF16,
                                             block_tables, context_lens, workspace,
                                             0 if workspace is None else workspace.nbytes, k_scale_cache, v_scale_cache,
                                             q_scale_cache, q_descale, k_descale, v_descale, p.scale, p.num_seqs,
                                             p.num_heads, p.num_kv_heads, p.head_dim, p.block_size,
                                             p.max_blocks_per_seq, p.num_blocks_total, p.window_size_left,
                                             _lib.launch_stream() if stream is None else stream)
        if rc:
            p.validate()  # (the same checks the call has just made: names the parameter set that failed)
            check(rc, "paged_decode_fp8")

    def quant_workspace_bytes(self) -> int:
        p = self.params
        return int(lib().rvllm_paged_decode_quant_workspace_size(p.num_seqs, p.num_heads, p.num_kv_heads, p.head_dim))

    def launch_quant(self, q_fp8, k_cache, v_cache, out_fp8, out_scale, round_dtype, block_tables, context_lens,
                     workspace, k_scale_cache=None, v_scale_cache=None, q_scale_cache=None, q_descale=None,
                     k_descale=None, v_descale=None, stream=None) -> None:
        """Attention + LSE combine + per-token FP8 quantisation of the [heads*head_dim] row in one call."""
        p = self.params
        rc = native().rvllm_paged_decode_fp8_quant(q_fp8, k_cache, v_cache, out_fp8, out_scale, round_dtype, block_tables,
                                                   context_lens, workspace, workspace.nbytes, k_scale_cache, v_scale_cache,
                                                   q_scale_cache, q_descale, k_descale, v_descale, p.scale, p.num_seqs,
                                                   p.num_heads, p.num_kv_heads, p.head_dim, p.block_size,
                                                   p.max_blocks_per_seq, p.num_blocks_total, p.window_size_left,
                                                   _lib.launch_stream() if stream is None else stream)
        if rc:
            p.validate()
            check(rc, "paged_decode_fp8_quant")
