"""All layers of a decode step of a few rows in one launch (csrc/decode_layers.cu).

`DecodeLayers.plan(...)` looks a model over: it is taken when every run of the schedule is the dense design's layer (RMSNorm,
grouped-query attention with a rotation of whole heads or none, RMSNorm, SwiGLU) of one set of sizes, in bfloat16, each
with a cache of its own. Any other model has no plan, and its layers run one by one. The plan holds the layers' descriptors
(addresses of weights, gains and caches, which live as long as the engine) on the device, and the words that the launch's
CTAs exchange, kept with their tags from step to step: a plan's steps follow one another on one stream, as an engine's do.
"""
from __future__ import annotations

import ctypes
from typing import Optional

import torch

from ..cache.pages import PAGE_TOKENS
from . import lib
from .attention_dispatch import _tc_fits
from .kernels import _chk
from .lib import KernelError, code, offer, ptr, stream_ptr

KERNEL_ROWS = 8         # rows that the kernel takes at most
# Rows up to which a step takes the one launch. 0: never.
MAX_ROWS = 8
# And rows times the widest product's columns: every CTA reads all of a product's rows, twice their size with the tags. One launch
# against the layers one by one, ms a step behind 200 positions with a vocabulary of 8,192: 0.6B shape (3,072 columns) 1 row
# 0.56 / 0.80, 3 rows 0.61 / 0.99, 8 rows 0.67 / 1.02; 4B shape's first 8 layers (9,728 columns) 1 row 0.45 / 0.70, 4 rows
# 0.47 / 0.57, 8 rows 0.51 / 0.59; 8B shape's first 6 layers (12,288 columns) 1 row 0.51 / 0.84, 4 rows 0.53 / 0.69; 4 layers of 5,120
# with 25,600 columns 1 row 0.74 / 1.24, 2 rows 0.75 / 1.27; 4 layers of 2,048 with 32,768 columns 2 rows 0.37 / 0.53.
MAX_ROW_COLUMNS = 8 * 9728
# And rows times the longest sequence's pages times kv heads (at least 8), by head size: behind long caches the page loop and the merge of the runs bound a
# layer, where the layers one by one stream pages with three CTAs an SM. ms a step, one launch / one by one, 0.6B shape: heads of 128,
# 8 rows x 250 pages 3.13 / 3.51, x 313 3.92 / 4.12, x 438 5.55 / 5.33, x 625 8.12 / 7.23; 4 rows x 625 3.99 / 4.35; 1 row x 625
# 1.70 / 2.23, x 1,016 2.46 / 3.03. Heads of 64, 8 rows x 250 2.62 / 2.70, x 625 6.98 / 5.26; 2 rows x 625 2.05 / 2.34. 12 layers of 32
# kv heads of 64, 8 rows x 33 0.89 / 1.07, x 64 1.30 / 1.20, x 250 4.82 / 2.88. Two kv heads, 8 rows x 250: 1.34 / 1.46. (Heads of
# 128 with more than 8 kv heads go by the same count and are not measured.)
MAX_PAGE_TILES = {64: 14336, 128: 23552}


def most_runs(pages: int) -> int:
    """Runs of pages that a sequence of at most so many is cut into at most: twos up to 16 pages, fours beyond (csrc/decode_layers.cu)."""
    return max(-(-min(pages, 16) // 2), -(-pages // 4) if pages > 16 else 0)


class DecodeLayers:
    # Tags that launches may use before the words are cleared and the tags begin again at 1: a tag names one stage of one launch as
    # long as 32 bits do not wrap (74 million steps of 28 layers, ten hours of steps of 0.5 ms).
    TAG_LIMIT = 2 ** 32 - 1
    # Looks at a word that has not come after which a wait is given up (a second and more).
    WAIT_LOOKS = 1 << 22

    def __init__(self, rows, sizes: dict, groups: list, device):
        self.host_table = torch.tensor(rows, dtype=torch.int64)                 # [layers, 12]
        self.table = self.host_table.to(device)
        self.sizes = sizes
        self.groups = groups                       # (K cache, V cache, window) of every storage group
        z = sizes
        self.words = torch.zeros((KERNEL_ROWS * (2 * (z["D"] + z["H"] * z["HD"] + z["F"]) + z["D"] + (z["H"] + 2 * z["KV"]) * z["HD"] // 2),),
                                 dtype=torch.int64, device=device)
        self.sync = torch.zeros((2,), dtype=torch.int32, device=device)
        self.part: Optional[torch.Tensor] = None
        self._retired: list[torch.Tensor] = []     # outgrown buffers stay alive: a captured graph may still hold their address
        self.declined = False                      # the launch's CTAs cannot all be resident here: the layers run one by one
        self._tags = 0                             # tags used since the words were cleared

    @classmethod
    def plan(cls, model, cache, runtime) -> Optional["DecodeLayers"]:
        from ..parts.attention import GQAttention
        from ..parts.block import PreNormResidual
        from ..parts.feedforward import SwiGLUDense
        from ..parts.norms import OffsetRMSNorm, RMSNorm
        from ..parts.position import NoPosition, RopeNeox
        if runtime.act_dtype != torch.bfloat16 or not model.schedule:
            return None
        rows, sizes, windows = [], None, {}
        for i, e in enumerate(model.schedule):
            block, view = model.layers[e.layer], cache.views[i]
            if type(block) is not PreNormResidual or block.mult != 1.0 or e.add_embedding or e.add_vector is not None or not view.writes:
                return None
            mix, ffn = block.mixer, block.ffn
            n1, n2 = block.norms.get("mixer"), block.norms.get("ffn")
            if type(mix) is not GQAttention or type(ffn) is not SwiGLUDense or ffn.out_dtype is not None:
                return None
            if type(n1) not in (RMSNorm, OffsetRMSNorm) or type(n2) not in (RMSNorm, OffsetRMSNorm) or n1.eps != n2.eps:
                return None
            if type(mix.position) not in (RopeNeox, NoPosition):
                return None
            cos, sin, rot = mix.position.fused_tables()
            if cos is not None and rot != mix.HD:
                return None
            qg, kg = mix.q_gain, mix.k_gain
            if (qg is None) != (kg is None) or (qg is not None and (qg.dtype != kg.dtype or qg.numel() != mix.HD or kg.numel() != mix.HD)):
                return None
            if n1.gain.dtype != n2.gain.dtype or n1.gain.numel() != mix.D or n2.gain.numel() != mix.D or ffn.D != mix.D:
                return None
            own = dict(D=mix.D, H=mix.H, KV=mix.KV, HD=mix.HD, F=ffn.F, eps=n1.eps, qk_eps=mix.qk_eps, gain_dtype=code(n1.gain.dtype),
                       qk_dtype=code(qg.dtype) if qg is not None else 0, cos=cos, sin=sin)
            if sizes is None:
                sizes = own
            elif any(own[k] is not sizes[k] if k in ("cos", "sin") else own[k] != sizes[k] for k in own):
                return None
            weights = [mix.w_qkv, mix.w_o, ffn.w_gate_up, ffn.w_down]
            shapes = [((mix.H + 2 * mix.KV) * mix.HD, mix.D), (mix.D, mix.H * mix.HD), (2 * ffn.F, mix.D), (mix.D, ffn.F)]
            if any(w.dtype != torch.bfloat16 or not w.is_contiguous() or tuple(w.shape) != s for w, s in zip(weights, shapes)):
                return None
            if windows.setdefault(view.group, mix.window or 0) != (mix.window or 0):
                return None
            k, v = view.k, view.v
            if v is None or k.dtype != torch.bfloat16 or v.dtype != k.dtype or k.shape != v.shape or tuple(k.shape[1:]) != (mix.KV, PAGE_TOKENS, mix.HD):
                return None
            row0, rest = divmod(k.data_ptr() - cache.keys[view.group].data_ptr(), mix.HD * 2)
            if rest or v.data_ptr() - cache.values[view.group].data_ptr() != row0 * mix.HD * 2:
                return None
            words = [t.data_ptr() if t is not None else 0 for t in [*weights, n1.gain, n2.gain, qg, kg, k, v]]
            if any(w % 16 for w in words):
                return None                        # (the copies and vector loads want 16-byte boundaries)
            rows.append(words + [row0, view.group])
        groups = [(cache.keys[g], cache.values[g], windows.get(g, 0)) for g in range(len(cache.keys))]
        if any(v is None or k.numel() // sizes["HD"] > 0x7fffffff for k, v, _ in groups):
            return None
        if not lib.load().mynah_decode_layers_supported(1, sizes["D"], sizes["H"], sizes["KV"], sizes["HD"], sizes["F"], len(rows), len(groups)):
            return None
        return cls(rows, sizes, groups, runtime.device)

    def takes(self, ctx) -> bool:
        z, rows = self.sizes, 1 << (ctx.T - 1).bit_length()          # (as a captured step pads them: both take the same route)
        if self.declined or not ctx.is_decode or rows > min(MAX_ROWS, KERNEL_ROWS) or rows * max(z["D"], z["H"] * z["HD"], z["F"]) > MAX_ROW_COLUMNS:
            return False
        # (Beyond what the tensor-core kernels' merge takes the layers one by one have the general kernel only: 4B shape's first 8
        # layers, 8 rows x 625 pages 2.80 / 12.75.)
        return rows * ctx.decode_splits * max(z["KV"], 8) <= MAX_PAGE_TILES[z["HD"]] or not _tc_fits(z["H"], z["KV"], ctx.decode_splits)

    def count_launch(self, layers: Optional[int] = None) -> None:
        """To be called before every launch, replayed ones too, on the launch's stream: keeps the tags from wrapping, after which
        words that were written long ago, or never, would pass for new ones."""
        n = 2 * (layers or self.table.shape[0]) + 2   # as the kernel moves its tags on
        if self._tags + n > self.TAG_LIMIT:
            for t in (self.sync, self.words, self.part, *self._retired):
                if t is not None:
                    t.zero_()
            self._tags = 0
        self._tags += n

    def _partials(self, rows: int, splits: int) -> torch.Tensor:
        need = rows * self.sizes["H"] * most_runs(splits) * (self.sizes["HD"] + 2)
        if self.part is None or self.part.numel() < need:
            if torch.cuda.is_current_stream_capturing():
                raise KernelError("decode_layers: the pages' partial results would have to grow during graph capture")
            if self.part is not None:
                self._retired.append(self.part)
                need = max(need, 2 * self.part.numel())          # (what has been outgrown is never more than what is in use)
            self.part = torch.zeros((need,), dtype=torch.int64, device=self.words.device)
        return self.part

    def forward(self, x: torch.Tensor, ctx, runtime, layers: Optional[range] = None) -> bool:
        """The residual stream x [T, D] (fp32, updated in place) behind all layers, or behind those of a range of them. A launch for
        every layer gives the bits that one for all of them gives: what is handed on from layer to layer is the stream. False:
        declined, nothing was done (where the process may use fewer SMs than the device has); `takes` says no from then on."""
        z, M, S = self.sizes, ctx.T, ctx.decode_splits
        layers = range(self.table.shape[0]) if layers is None else layers
        _chk(x, "residual", torch.float32, 2)
        if tuple(x.shape) != (M, z["D"]):
            raise KernelError(f"decode_layers: the residual is {tuple(x.shape)}, the step has {(M, z['D'])}")
        words = []
        for (k, v, window), p in zip(self.groups, ctx.pages):
            words += [k.data_ptr(), v.data_ptr(), k.numel() // z["HD"], window, p.indptr.data_ptr(), p.ids.data_ptr(), p.base.data_ptr(), p.n_pages]
        cos, sin = z["cos"], z["sin"]
        if not torch.cuda.is_current_stream_capturing():
            self.count_launch(len(layers))         # (a recorded launch counts when it is replayed)
        part = self._partials(M, S)
        self.declined = not offer(
            "mynah_decode_layers", ptr(self.table[layers.start]), ptr(self.host_table[layers.start]), len(layers),
            M, z["D"], z["H"], z["KV"], z["HD"], z["F"], S, ptr(x), ptr(self.words), ptr(part), part.numel(), ptr(self.sync),
            z["gain_dtype"], z["eps"], z["qk_dtype"], z["qk_eps"], ptr(cos), ptr(sin), cos.shape[0] if cos is not None else 0,
            ptr(ctx.kv_len), len(self.groups), (ctypes.c_longlong * len(words))(*words), ptr(ctx.status), runtime.sm_count, self.WAIT_LOOKS,
            stream_ptr())
        if self.declined and layers.start > 0:
            raise KernelError("decode_layers: declined behind the first layers of a step")
        return not self.declined
