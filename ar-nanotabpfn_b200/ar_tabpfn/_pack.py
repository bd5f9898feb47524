"""Pack module weights into the flat fp32 device buffer the kernels read.

All matrices are stored transposed ([in][out]); the feature-attention pair
(out_proj, v_proj) is folded into one [D][D] matrix because that attention runs
over a single token (ar_tabpfn/model/inference.py:771-773 of the reference:
softmax over one key is 1, so the block equals out_proj(v_proj(x)) and the q/k
projections never influence the result).
"""
from __future__ import annotations

import ctypes as C
from typing import List, Tuple

import torch

from . import _lib

_ALIGN = 64  # floats


def _split_bf16(w: torch.Tensor):
    """fp64 matrix -> (hi, lo) bf16 parts with hi + lo ~= w to 16 mantissa bits."""
    hi = w.to(torch.float32).to(torch.bfloat16)
    lo = (w - hi.to(torch.float64)).to(torch.float32).to(torch.bfloat16)
    return hi, lo


def _swizzle(blocks: torch.Tensor) -> torch.Tensor:
    """[..., rows][64] bf16 -> the 128-byte-swizzled K-major shared-memory image of every [rows][64] block:
    16-byte chunk c of row r is stored at chunk position c ^ (r % 8)."""
    r = torch.arange(8)[:, None]
    return blocks.reshape(-1, 8, 8, 8)[:, r, torch.arange(8)[None, :] ^ r].reshape(-1)


def tile_weight(hi: torch.Tensor, lo: torch.Tensor, mode: str, force_lo: bool = False):
    """Tile the hi and lo part of an nn.Linear weight [N][K] for the tensor-core chain.

    The result is the exact byte stream the kernel's weight ring consumes: a sequence of
    slabs, each a stack of swizzled [rows][64 k] blocks, hi part then (optionally) lo part.
      mode "full":   one slab per 64-wide k-chunk holding all N rows            (N = d_model)
      mode "ntile":  per 128-row output tile one 16 KB slab per k-chunk         (hidden GEMMs)
    Returns (flat bf16 tensor, has_lo)."""
    N, K = hi.shape
    assert K % 64 == 0
    has_lo = force_lo or bool((lo != 0).any())
    parts = torch.stack((hi, lo) if has_lo else (hi,))
    if mode == "full":
        return _swizzle(parts.reshape(-1, N, K // 64, 64).permute(2, 0, 1, 3)), has_lo
    assert N % 128 == 0
    return _swizzle(parts.reshape(-1, N // 128, 128, K // 64, 64).permute(1, 0, 3, 2, 4)), has_lo


class PackedModel:
    """All packing arithmetic (transposes, the fold of the feature attention, hi / lo splits,
    swizzled tiles) runs on the host in fp64, once per model version, and no packing kernels on the device.
    Each layout is made when the first call needs it (``prepare``, ``prepare_sequence``): new weights cost a
    call only what it reads."""

    def __init__(self, embedder, backbone, head, ar_tokens, device: torch.device):
        target, device = device, torch.device("cpu")
        layers = list(backbone.layers)
        attn0 = layers[0].attn_rows
        self.d_model = int(backbone.norm.weight.numel())
        self.n_heads = int(attn0.n_heads)
        self.head_dim = int(attn0.head_dim)
        self.d_ff = int(layers[0].ff[0].weight.shape[0])
        self.n_layers = len(layers)
        self.n_comp = int(head.num_components)
        self.n_ar = int(ar_tokens.shape[0])
        if int(head.dim_y) != 1:
            raise ValueError("only dim_y = 1 is supported")
        if int(head.head[0].weight.shape[0]) != self.d_ff:
            raise ValueError("head hidden width must equal d_ff")

        items: List[Tuple[str, torch.Tensor]] = []

        def add(name, t):
            items.append((name, t.detach().to(device=device, dtype=torch.float64).contiguous()))

        def T(w):  # nn.Linear weight [out][in] -> [in][out]
            return w.detach().to(device=device, dtype=torch.float64).t().contiguous()

        e = embedder
        add("wx", e.x_embed.weight[:, 0]); add("bx", e.x_embed.bias)
        add("wy", e.y_embed.weight[:, 0]); add("by", e.y_embed.bias)
        add("marker", e.marker_embed.weight); add("ar_tokens", ar_tokens)
        add("lnf_g", backbone.norm.weight); add("lnf_b", backbone.norm.bias)
        add("wa_t", T(head.head[0].weight)); add("ba", head.head[0].bias)
        add("wb_t", T(head.head[2].weight)); add("bb", head.head[2].bias)
        add("mean_bias", head.mean_bias); add("std_bias", head.std_bias); add("weight_bias", head.weight_bias)
        for i, l in enumerate(layers):
            wv = l.attn_features.v_proj.weight.detach().to(device=device, dtype=torch.float64)
            wo = l.attn_features.out_proj.weight.detach().to(device=device, dtype=torch.float64)
            add(f"{i}.wf_t", (wo @ wv).t())
            add(f"{i}.ln1_g", l.norm1.weight); add(f"{i}.ln1_b", l.norm1.bias)
            r = l.attn_rows
            add(f"{i}.wqkv_t", torch.cat([T(r.q_proj.weight), T(r.k_proj.weight), T(r.v_proj.weight)], dim=1))
            add(f"{i}.wo_t", T(r.out_proj.weight))
            add(f"{i}.ln2_g", l.norm2.weight); add(f"{i}.ln2_b", l.norm2.bias)
            add(f"{i}.w1_t", T(l.ff[0].weight)); add(f"{i}.b1", l.ff[0].bias)
            add(f"{i}.w2_t", T(l.ff[2].weight)); add(f"{i}.b2", l.ff[2].bias)
            add(f"{i}.ln3_g", l.norm3.weight); add(f"{i}.ln3_b", l.norm3.bias)

        offsets, total = {}, 0
        for name, t in items:
            offsets[name] = total
            total += (t.numel() + _ALIGN - 1) // _ALIGN * _ALIGN
        flat = torch.zeros(total, dtype=torch.float32, device=device)
        for name, t in items:
            flat[offsets[name]:offsets[name] + t.numel()] = t.reshape(-1).to(torch.float32)
        flat = flat.to(target)
        self.flat = flat
        base = flat.data_ptr()

        def P(name):
            return C.c_void_p(base + 4 * offsets[name])

        self._layers = (_lib.LayerWeights * self.n_layers)()
        for i in range(self.n_layers):
            for f, _ in _lib.LayerWeights._fields_:
                if not f.startswith(("tc_", "fma_", "mma_")):
                    setattr(self._layers[i], f, P(f"{i}.{f}"))
        m = _lib.Model()
        m.d_model, m.n_heads, m.head_dim, m.d_ff = self.d_model, self.n_heads, self.head_dim, self.d_ff
        m.n_layers, m.n_comp, m.n_ar_tokens = self.n_layers, self.n_comp, self.n_ar
        for f in ("wx", "bx", "wy", "by", "marker", "ar_tokens", "lnf_g", "lnf_b", "wa_t", "ba", "wb_t", "bb",
                  "mean_bias", "std_bias", "weight_bias"):
            setattr(m, f, P(f))
        m.layers = C.cast(self._layers, C.POINTER(_lib.LayerWeights))
        self.struct = m
        self.tc_flat = self.seq_flat = self.fma_flat = self.mma_flat = None
        self._w = dict(items)
        self._target = target
        self._made = set()
        self._split = {}
        D, Dff, H = self.d_model, self.d_ff, self.n_heads
        ranks = max(c for c in range(1, 9) if H % c == 0)
        if D % 64 == 0 and Dff % ranks == 0 and D // ranks % 16 == 0 and Dff // ranks % 32 == 0:
            m.seq_ranks = ranks      # what artab_sequence_workspace goes by; the stream itself: prepare_sequence

    def _once(self, name: str, make) -> None:
        if name not in self._made:
            make(self._w, self._target)
            self._made.add(name)

    def _halves(self, name: str):
        """bf16 hi and lo part of a matrix ("wb16": head.2 with 16 output columns), split all together once."""
        if not self._split:
            names = [n for n in self._w if n.endswith(("wf_t", "wqkv_t", "wo_t", "w1_t", "w2_t", "wa_t"))] + ["wb16"]
            wb = torch.zeros(self.d_ff, 16, dtype=torch.float64)
            wb[:, :3 * self.n_comp] = self._w["wb_t"]
            mats = [self._w[n] if n != "wb16" else wb for n in names]
            hi, lo = _split_bf16(torch.cat([m.reshape(-1) for m in mats]))
            for n, m, h, l in zip(names, mats, hi.split([m.numel() for m in mats]), lo.split([m.numel() for m in mats])):
                self._split[n] = h.view(m.shape), l.view(m.shape)
        return self._split[name]

    def prepare(self, bf16: bool) -> "PackedModel":
        """Lay the weights out for the dense chains of this precision."""
        if bf16:
            self._once("tensor_core", self._pack_tensor_core)
        if bf16 and self.tc_flat is not None:
            self._once("fragments", self._pack_fragments)
            self._split = {}
        else:
            self._once("panels", self._pack_panels)
        return self

    def prepare_sequence(self) -> None:
        """Lay the weights out for artab_decode_sequence."""
        if self.struct.seq_ranks:
            self._once("sequence", self._pack_sequence)

    def _pack_tensor_core(self, w, target):
        """bf16 hi/lo tiles for the tcgen05 per-token chain (d_model in {64,128,192}, d_ff % 128 == 0,
        3K <= 16).  Other shapes keep the fp32 FMA chain (the tc_* pointers stay NULL)."""
        D, Dff = self.d_model, self.d_ff
        device = torch.device("cpu")
        if D not in (64, 128, 192) or Dff % 128 != 0 or Dff > 1024 or 3 * self.n_comp > 16:
            return
        items = []

        def add(name, parts, mode, force_lo=False):   # parts: hi, lo [in][out]
            flat, has_lo = tile_weight(parts[0].t(), parts[1].t(), mode, force_lo)
            items.append((name, flat))
            return has_lo

        layer_lo = []
        for i in range(self.n_layers):
            bits = 0
            bits |= 1 * add(f"{i}.tc_wo", self._halves(f"{i}.wo_t"), "full")
            bits |= 2 * add(f"{i}.tc_w1", self._halves(f"{i}.w1_t"), "ntile")
            bits |= 4 * add(f"{i}.tc_w2", self._halves(f"{i}.w2_t"), "full")
            bits |= 8 * add(f"{i}.tc_wf", self._halves(f"{i}.wf_t"), "full")
            # q, k, v must agree on the lo part: they share one flag
            hi, lo = self._halves(f"{i}.wqkv_t")
            qkv_lo = bool((lo != 0).any())
            for j, nm in enumerate("qkv"):
                add(f"{i}.tc_w{nm}", (hi[:, j * D:(j + 1) * D], lo[:, j * D:(j + 1) * D]), "full", force_lo=qkv_lo)
            bits |= 16 * qkv_lo
            layer_lo.append(bits)
        head_bits = 1 * add("tc_wa", self._halves("wa_t"), "ntile")
        head_bits |= 2 * add("tc_wb", self._halves("wb16"), "full")
        offs, tot = {}, 0
        for name, t in items:
            offs[name] = tot
            tot += (t.numel() + 511) // 512 * 512          # 1 KiB alignment of every matrix
        flat = torch.zeros(tot, dtype=torch.bfloat16, device=device)
        for name, t in items:
            flat[offs[name]:offs[name] + t.numel()] = t
        flat = flat.to(target)
        self.tc_flat = flat
        base = flat.data_ptr()
        for i in range(self.n_layers):
            lw = self._layers[i]
            lw.tc_wo = base + 2 * offs[f"{i}.tc_wo"]
            lw.tc_w1 = base + 2 * offs[f"{i}.tc_w1"]
            lw.tc_w2 = base + 2 * offs[f"{i}.tc_w2"]
            lw.tc_wf = base + 2 * offs[f"{i}.tc_wf"]
            lw.tc_wqkv = base + 2 * offs[f"{i}.tc_wq"]
            lw.tc_lo = layer_lo[i]
        self.struct.tc_wa = base + 2 * offs["tc_wa"]
        self.struct.tc_wb = base + 2 * offs["tc_wb"]
        self.struct.tc_head_lo = head_bits

    def _pack_sequence(self, w, target):
        """Weight streams of the whole-sequence decode: per cluster rank the slices of every matrix in the
        order of use (layer by layer: fold, Q|K|V of the rank's heads | out-projection, MLP; then the head).
        A slice [K][N] is a sequence of units of 32 k x 16 columns, k blocks outermost; inside a unit element
        (k = 4s + e, n = 4g + c) sits at [c][s][g][e].  ``w`` holds the matrices as [in][out]."""
        D, Dff, K = self.d_model, self.d_ff, self.n_comp
        ranks = self.struct.seq_ranks
        hs, L = Dff // ranks, self.n_layers
        wb = torch.zeros(Dff, (3 * K + 15) // 16 * 16, dtype=torch.float64)
        wb[:, :3 * K] = w["wb_t"]
        f32 = lambda m: m.to(torch.float32)
        # -> [rank][units of its slice]
        cols = lambda m: (f32(m).reshape(m.shape[0] // 32, 8, 4, ranks, m.shape[1] // ranks // 16, 4, 4)
                          .permute(3, 0, 4, 6, 1, 5, 2).reshape(ranks, -1))
        rows = lambda m: f32(m).reshape(ranks, hs // 32, 8, 4, m.shape[1] // 16, 4, 4).permute(0, 1, 4, 6, 2, 5, 3).reshape(ranks, -1)
        by_rank = lambda m: m.reshape(D, 3, ranks, D // ranks).transpose(1, 2).reshape(D, 3 * D)   # q | k | v of a rank together
        mats = []
        for i in range(L):
            mats += [cols(w[f"{i}.wf_t"]), cols(by_rank(w[f"{i}.wqkv_t"]))]
            mats += [cols(w[f"{i}.wo_t"]), cols(w[f"{i}.w1_t"]), rows(w[f"{i}.w2_t"])]
        mats += [cols(w["wa_t"]), rows(wb)]
        self.struct.seq_vec_off = 4 * sum(m.shape[1] for m in mats)
        # after the matrices: per layer LayerNorm 1 / 2 vectors, b2, LayerNorm 3 vectors, b1 slice; final
        # LayerNorm, first bias of the head (slice)
        whole = lambda v: f32(v).reshape(1, -1).expand(ranks, -1)
        part = lambda v: f32(v).reshape(ranks, hs)
        for i in range(L):
            mats += [whole(w[f"{i}.{k}"]) for k in ("ln1_g", "ln1_b", "ln2_g", "ln2_b", "b2", "ln3_g", "ln3_b")] + [part(w[f"{i}.b1"])]
        mats += [whole(w["lnf_g"]), whole(w["lnf_b"]), part(w["ba"])]
        flat = torch.cat(mats, dim=1)
        self.struct.seq_rank_bytes = 4 * flat.shape[1]
        self.seq_flat = flat.to(target)
        self.struct.seq_w = self.seq_flat.data_ptr()

    def _pack_panels(self, w, target):
        """D x D panels of every matrix for the register-tiled fp32 chain, in the order it uses them."""
        D, Dff, K = self.d_model, self.d_ff, self.n_comp
        if D not in (64, 128, 192) or Dff % D or Dff > 1024 or 3 * K > D:
            return
        chunks = range(0, Dff, D)
        wb = torch.zeros(Dff, D, dtype=torch.float64)
        wb[:, :3 * K] = w["wb_t"]
        stacks = []
        for i in range(self.n_layers):
            stacks.append([w[f"{i}.wf_t"], *w[f"{i}.wqkv_t"].split(D, dim=1)])
            stacks.append([w[f"{i}.wo_t"]] + [p for j in chunks for p in (w[f"{i}.w1_t"][:, j:j + D], w[f"{i}.w2_t"][j:j + D])])
        stacks.append([p for j in chunks for p in (w["wa_t"][:, j:j + D], wb[j:j + D])])
        flat = torch.cat([p.reshape(-1).to(torch.float32) for st in stacks for p in st]).to(target)
        self.fma_flat = flat
        at = flat.data_ptr()
        for n, st in enumerate(stacks):
            if n == len(stacks) - 1:
                self.struct.fma_head = at
            else:
                setattr(self._layers[n // 2], ("fma_pre", "fma_post")[n % 2], at)
            at += 4 * D * D * len(st)

    def _pack_fragments(self, w, target):
        """mma.m16n8k16 B fragments for the few-row bf16 chain: four slices of every matrix (by output column, w2 and
        head.2 by input row), hi part then lo part.  A part is a sequence of units of 8 columns x 32 k, k innermost;
        in a unit lane (g, t) holds column g, k = 16 ks + 8 half + 2 t + e at [ks][half][e]."""
        D, Dff, K = self.d_model, self.d_ff, self.n_comp
        hs = Dff // 4

        # -> the hi and the lo part, each [rank][fragment order]
        def cols(name):
            ms = self._halves(name)
            if name.endswith("wqkv_t"):   # q | k | v of a rank together
                ms = [m.reshape(D, 3, 4, D // 4).transpose(1, 2).reshape(D, 3 * D) for m in ms]
            k, n = ms[0].shape
            return [m.reshape(k // 32, 2, 2, 4, 2, 4, n // 32, 8).permute(5, 6, 0, 7, 3, 1, 2, 4).reshape(4, -1) for m in ms]

        def rows(name):
            ms = self._halves(name)
            return [m.reshape(4, hs // 32, 2, 2, 4, 2, m.shape[1] // 8, 8).permute(0, 6, 1, 7, 4, 2, 3, 5).reshape(4, -1) for m in ms]

        streams = lambda *parts: torch.cat(sum(parts, []), dim=1).reshape(-1)
        stacks = []
        for i in range(self.n_layers):
            stacks.append(streams(cols(f"{i}.wf_t"), cols(f"{i}.wqkv_t")))
            stacks.append(streams(cols(f"{i}.wo_t"), cols(f"{i}.w1_t"), rows(f"{i}.w2_t")))
        stacks.append(streams(cols("wa_t"), rows("wb16")))
        self.mma_flat = torch.cat(stacks).to(target)
        at = self.mma_flat.data_ptr()
        for n, st in enumerate(stacks):
            if n == len(stacks) - 1:
                self.struct.mma_head = at
            else:
                setattr(self._layers[n // 2], ("mma_pre", "mma_post")[n % 2], at)
            at += 2 * st.numel()

    @property
    def ref(self):
        return C.byref(self.struct)


def packed_for(owner, embedder, backbone, head, ar_tokens, device) -> PackedModel:
    """Cache the packed weights on `owner`, keyed by device and parameter versions."""
    params = [ar_tokens] + list(embedder.parameters()) + list(backbone.parameters()) + list(head.parameters())
    key = (str(device),) + tuple((p.data_ptr(), p._version) for p in params)
    cached = getattr(owner, "_artab_packed", None)
    if cached is None or cached[0] != key:
        cached = (key, PackedModel(embedder, backbone, head, ar_tokens, device))
        owner._artab_packed = cached
    return cached[1]
