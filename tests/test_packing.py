"""Weight layouts for the kernels: every element where the layout's definition puts it, and no layout before a call
needs it.  Runs on the host."""
import random

import pytest
import torch

from ar_tabpfn import ARTabPFN
from ar_tabpfn._pack import PackedModel

CONFIGS = [dict(d_model=192, n_heads=6, n_layers=2, d_ff=768, num_components=5),
           dict(d_model=64, n_heads=4, n_layers=2, d_ff=128, num_components=3),
           dict(d_model=128, n_heads=8, n_layers=1, d_ff=512, num_components=5)]


def _packed(cfg):
    torch.manual_seed(0)
    m = ARTabPFN(num_features=3, **cfg)
    return PackedModel(m.embedder, m.backbone, m.head, m.ar_tokens, torch.device("cpu"))


def _split(x):
    hi = x.float().bfloat16()
    return hi, (x - hi.double()).float().bfloat16()


def _places(K, N, n=60):
    rng = random.Random(K * 1000 + N)
    return [(rng.randrange(K), rng.randrange(N)) for _ in range(n)] + [(0, 0), (K - 1, N - 1)]


def _matrices(p):
    """[in][out] in the order of use: per layer fold, q | k | v, out-projection, W1, W2; then the head."""
    w = p._w
    for i in range(p.n_layers):
        yield from ((f"{i}.{n}", w[f"{i}.{n}"]) for n in ("wf_t", "wqkv_t", "wo_t", "w1_t", "w2_t"))
    yield "wa_t", w["wa_t"]
    wb = torch.zeros(p.d_ff, 16, dtype=torch.float64)
    wb[:, :3 * p.n_comp] = w["wb_t"]
    yield "wb_t", wb


def _slice(name, m, r, ranks):
    if name.endswith(("w2_t", "wb_t")):
        return m.chunk(ranks, dim=0)[r]
    if name.endswith("wqkv_t"):
        return torch.cat([q.chunk(ranks, dim=1)[r] for q in m.chunk(3, dim=1)], dim=1)
    return m.chunk(ranks, dim=1)[r]


@pytest.mark.parametrize("cfg", CONFIGS, ids=lambda c: "d%d" % c["d_model"])
def test_sequence_stream(cfg):
    p = _packed(cfg)
    p.prepare_sequence()
    ranks = p.struct.seq_ranks
    for r in range(ranks):
        flat, at = p.seq_flat[r], 0
        for name, m in _matrices(p):
            s = _slice(name, m, r, ranks)
            K, N = s.shape
            for k, n in _places(K, N):
                unit = (k // 32) * (N // 16) + n // 16
                inside = ((n % 4 * 8 + k % 32 // 4) * 4 + n % 16 // 4) * 4 + k % 4
                assert flat[at + unit * 512 + inside] == s[k, n].float(), (name, k, n)
            at += K * N
        assert p.struct.seq_vec_off == 4 * at
        assert torch.equal(flat[at:at + p.d_model], p._w["0.ln1_g"].float())


@pytest.mark.parametrize("cfg", CONFIGS, ids=lambda c: "d%d" % c["d_model"])
def test_fragments(cfg):
    p = _packed(cfg).prepare(bf16=True)
    mats, at = dict(_matrices(p)), 0
    groups = [g for i in range(p.n_layers) for g in ((f"{i}.wf_t", f"{i}.wqkv_t"), (f"{i}.wo_t", f"{i}.w1_t", f"{i}.w2_t"))]
    for group in groups + [("wa_t", "wb_t")]:
        for r in range(4):
            for name in group:
                s = _slice(name, mats[name], r, 4)
                K, N = s.shape
                for part in _split(s):
                    for k, n in _places(K, N):
                        unit = (n // 8) * (K // 32) + k // 32
                        ks, half, t, e = k % 32 // 16, k % 16 // 8, k % 8 // 2, k % 2
                        assert p.mma_flat[at + unit * 256 + (n % 8 * 4 + t) * 8 + ks * 4 + half * 2 + e] == part[k, n], (name, k, n)
                    at += K * N
    assert at == p.mma_flat.numel()


@pytest.mark.parametrize("cfg", CONFIGS, ids=lambda c: "d%d" % c["d_model"])
def test_tiles(cfg):
    p = _packed(cfg).prepare(bf16=True)
    at = (p._layers[0].tc_w1 - p.tc_flat.data_ptr()) // 2, (p._layers[0].tc_w2 - p.tc_flat.data_ptr()) // 2
    for start, name, rows in ((at[0], "0.w1_t", 128), (at[1], "0.w2_t", p.d_model)):
        w = p._w[name].t()          # [N][K]
        N, K = w.shape
        for part, half in enumerate(_split(w)):
            for n, k in _places(N, K):
                j, kc, row, chunk = n // rows, k // 64, n % rows, k % 64 // 8
                block = (j * 2 + part) * (K // 64) + kc if rows == 128 and name.endswith("w1_t") else kc * 2 + part
                assert p.tc_flat[start + (block * rows + row) * 64 + (chunk ^ row % 8) * 8 + k % 8] == half[n, k], (name, n, k)


def test_a_layout_is_made_when_a_call_needs_it():
    layouts = lambda p: [getattr(p, n) is not None for n in ("tc_flat", "mma_flat", "fma_flat", "seq_flat")]
    p = _packed(CONFIGS[1])
    assert layouts(p) == [False] * 4 and p.struct.seq_ranks == 4 and not p.struct.seq_w
    assert layouts(p.prepare(bf16=False)) == [False, False, True, False]
    flat = p.fma_flat
    assert layouts(p.prepare(bf16=True)) == [True, True, True, False] and p.prepare(bf16=False).fma_flat is flat
    p.prepare_sequence()
    assert layouts(p) == [True] * 4
    q = _packed(dict(d_model=64, n_heads=4, n_layers=1, d_ff=128, num_components=20))   # outside the tensor-core chain
    assert layouts(q.prepare(bf16=True)) == [False, False, True, False]
