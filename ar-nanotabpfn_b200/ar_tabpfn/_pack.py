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


def _swizzle_block(blk: torch.Tensor) -> torch.Tensor:
    """[rows][64] bf16 -> the 128-byte-swizzled K-major shared-memory image of that block:
    16-byte chunk c of row r is stored at chunk position c ^ (r % 8)."""
    rows = blk.shape[0]
    chunks = blk.reshape(rows, 8, 8)
    pos = torch.arange(8, device=blk.device)[None, :] ^ (torch.arange(rows, device=blk.device)[:, None] % 8)
    out = torch.empty_like(chunks)
    out.scatter_(1, pos[:, :, None].expand(rows, 8, 8), chunks)
    return out.reshape(-1)


def tile_weight(w: torch.Tensor, mode: str, force_lo: bool = False):
    """Tile an nn.Linear weight [N][K] (fp64) for the tensor-core chain.

    The result is the exact byte stream the kernel's weight ring consumes: a sequence of
    slabs, each a stack of swizzled [rows][64 k] blocks, hi part then (optionally) lo part.
      mode "full":   one slab per 64-wide k-chunk holding all N rows            (N = d_model)
      mode "ntile":  per 128-row output tile one 16 KB slab per k-chunk         (hidden GEMMs)
    Returns (flat bf16 tensor, has_lo)."""
    N, K = w.shape
    assert K % 64 == 0
    hi, lo = _split_bf16(w)
    has_lo = force_lo or bool((lo != 0).any())
    slabs = []
    if mode == "full":
        for kc in range(K // 64):
            for part in ((hi, lo) if has_lo else (hi,)):
                slabs.append(_swizzle_block(part[:, kc * 64:(kc + 1) * 64].contiguous()))
    else:
        assert N % 128 == 0
        for j in range(N // 128):
            for part in ((hi, lo) if has_lo else (hi,)):
                for kc in range(K // 64):
                    slabs.append(_swizzle_block(part[j * 128:(j + 1) * 128, kc * 64:(kc + 1) * 64].contiguous()))
    return torch.cat(slabs), has_lo


class PackedModel:
    """All packing arithmetic (transposes, the fold of the feature attention, hi / lo splits,
    swizzled tiles) runs on the host in fp64, once per model version; the device sees two copies
    (the fp32 buffer and the bf16 tile stream) and no packing kernels."""

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
        self._pack_tensor_core(embedder, backbone, head, target)
        self._pack_sequence(dict(items), target)
        self._pack_panels(dict(items), target)
        self._pack_fragments(dict(items), target)

    def _pack_tensor_core(self, embedder, backbone, head, target):
        """bf16 hi/lo tiles for the tcgen05 per-token chain (d_model in {64,128,192}, d_ff % 128 == 0,
        3K <= 16).  Other shapes keep the fp32 FMA chain (the tc_* pointers stay NULL)."""
        D, Dff = self.d_model, self.d_ff
        device = torch.device("cpu")
        self.tc_flat = None
        if D not in (64, 128, 192) or Dff % 128 != 0 or Dff > 1024 or 3 * self.n_comp > 16:
            return
        f64 = lambda t: t.detach().to(device=device, dtype=torch.float64)
        items = []

        def add(name, w, mode, force_lo=False):
            flat, has_lo = tile_weight(w, mode, force_lo)
            items.append((name, flat))
            return has_lo

        layer_lo = []
        for i, l in enumerate(backbone.layers):
            r = l.attn_rows
            bits = 0
            bits |= 1 * add(f"{i}.tc_wo", f64(r.out_proj.weight), "full")
            bits |= 2 * add(f"{i}.tc_w1", f64(l.ff[0].weight), "ntile")
            bits |= 4 * add(f"{i}.tc_w2", f64(l.ff[2].weight), "full")
            wf = f64(l.attn_features.out_proj.weight) @ f64(l.attn_features.v_proj.weight)
            bits |= 8 * add(f"{i}.tc_wf", wf, "full")
            # q, k, v must agree on the lo part: they share one flag
            qkv_lo = any(bool((_split_bf16(f64(p.weight))[1] != 0).any()) for p in (r.q_proj, r.k_proj, r.v_proj))
            for nm, p in (("q", r.q_proj), ("k", r.k_proj), ("v", r.v_proj)):
                add(f"{i}.tc_w{nm}", f64(p.weight), "full", force_lo=qkv_lo)
            bits |= 16 * qkv_lo
            layer_lo.append(bits)
        head_bits = 1 * add("tc_wa", f64(head.head[0].weight), "ntile")
        wb = torch.zeros(16, Dff, dtype=torch.float64, device=device)
        wb[: 3 * self.n_comp] = f64(head.head[2].weight)
        head_bits |= 2 * add("tc_wb", wb, "full")
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
        D, Dff, H, Dh, K = self.d_model, self.d_ff, self.n_heads, self.head_dim, self.n_comp
        ranks = max(c for c in range(1, 9) if H % c == 0)
        self.seq_flat = None
        if D % 64 or Dff % ranks or D // ranks % 16 or Dff // ranks % 32:
            return
        ds, hs, qs = D // ranks, Dff // ranks, H // ranks * Dh
        wb = torch.zeros(Dff, (3 * K + 15) // 16 * 16, dtype=torch.float64)
        wb[:, :3 * K] = w["wb_t"]
        unit = lambda m: (m.reshape(m.shape[0] // 32, 8, 4, m.shape[1] // 16, 4, 4).permute(0, 3, 5, 1, 4, 2)
                          .to(torch.float32).reshape(-1))
        streams = []
        for r in range(ranks):
            cols = lambda m, n: m[:, r * n:(r + 1) * n]
            parts = []

            def pre(i):
                parts.append(cols(w[f"{i}.wf_t"], ds))
                parts.append(torch.cat([cols(m, qs) for m in w[f"{i}.wqkv_t"].split(D, dim=1)], dim=1))

            pre(0)
            for i in range(self.n_layers):
                parts += [cols(w[f"{i}.wo_t"], ds), cols(w[f"{i}.w1_t"], hs), w[f"{i}.w2_t"][r * hs:(r + 1) * hs]]
                if i + 1 < self.n_layers:
                    pre(i + 1)
            parts += [cols(w["wa_t"], hs), wb[r * hs:(r + 1) * hs]]
            # after the matrices: per layer LayerNorm 1 / 2 vectors, b2, LayerNorm 3 vectors, b1 slice; final
            # LayerNorm, first bias of the head (slice)
            part = lambda v: v[r * hs:(r + 1) * hs]
            vec = []
            for i in range(self.n_layers):
                vec += [w[f"{i}.{k}"] for k in ("ln1_g", "ln1_b", "ln2_g", "ln2_b", "b2", "ln3_g", "ln3_b")] + [part(w[f"{i}.b1"])]
            vec += [w["lnf_g"], w["lnf_b"], part(w["ba"])]
            mats = [unit(p) for p in parts]
            self.struct.seq_vec_off = 4 * sum(m.numel() for m in mats)
            streams.append(torch.cat(mats + [v.reshape(-1).to(torch.float32) for v in vec]))
        flat = torch.stack(streams)
        self.struct.seq_ranks = ranks
        self.struct.seq_rank_bytes = 4 * flat.shape[1]
        self.seq_flat = flat.to(target)
        self.struct.seq_w = self.seq_flat.data_ptr()

    def _pack_panels(self, w, target):
        """D x D panels of every matrix for the register-tiled fp32 chain, in the order it uses them."""
        D, Dff, K = self.d_model, self.d_ff, self.n_comp
        self.fma_flat = None
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
        self.mma_flat = None
        if self.tc_flat is None:
            return
        D, Dff, K = self.d_model, self.d_ff, self.n_comp
        ds, hs = D // 4, Dff // 4
        wb = torch.zeros(Dff, 16, dtype=torch.float64)
        wb[:, :3 * K] = w["wb_t"]

        def parts(m):
            u = lambda t: t.reshape(m.shape[0] // 32, 2, 2, 4, 2, m.shape[1] // 8, 8).permute(5, 0, 6, 3, 1, 2, 4).reshape(-1)
            hi, lo = _split_bf16(m)
            return [u(hi.to(torch.bfloat16)), u(lo.to(torch.bfloat16))]

        def streams(matrices):
            return torch.cat([p for r in range(4) for m in matrices(r) for p in parts(m.contiguous())])

        cols = lambda m, r: m[:, r * m.shape[1] // 4:(r + 1) * m.shape[1] // 4]
        rows = lambda m, r: m[r * hs:(r + 1) * hs]
        stacks = []
        for i in range(self.n_layers):
            stacks.append(streams(lambda r: [cols(w[f"{i}.wf_t"], r), torch.cat([cols(m, r) for m in w[f"{i}.wqkv_t"].split(D, dim=1)], dim=1)]))
            stacks.append(streams(lambda r: [cols(w[f"{i}.wo_t"], r), cols(w[f"{i}.w1_t"], r), rows(w[f"{i}.w2_t"], r)]))
        stacks.append(streams(lambda r: [cols(w["wa_t"], r), rows(wb, r)]))
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
