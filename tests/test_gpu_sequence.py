"""The one-launch decode of a whole sampling job against the CPU oracle: every kernel variant (streams per
cluster, head size, cache type, shared or own contexts) at the sizes where its tiles end: context tiles of
32 keys, private keys of 32 in four parts, clusters with a stream missing, several heads per CTA.  Every case says
whether the one-launch path is to take it."""
import ctypes

import pytest
import torch

import artab_oracle as orc

pytestmark = pytest.mark.gpu

# d_model, heads, layers, d_ff, components, streams, context rows, targets, shared; one launch in fp32, in bf16
CASES = [
    (64, 4, 2, 128, 5, 1, 1, 3, True, True, True),          # one key, one stream
    (64, 4, 1, 128, 20, 5, 33, 6, True, True, True),        # head size 16, twenty components
    (64, 2, 1, 128, 5, 37, 31, 4, True, True, True),        # two CTAs per cluster, context one key short of a tile
    (64, 1, 1, 64, 5, 3, 64, 5, True, False, False),        # one head: no cluster to form
    (128, 4, 2, 256, 5, 130, 40, 4, True, True, True),      # four streams per cluster, the last cluster not full
    (128, 2, 1, 256, 3, 9, 70, 5, False, True, True),       # head size 64, own contexts
    (128, 8, 1, 512, 5, 200, 30, 3, True, False, False),    # eight CTAs, more streams than one wave
    (192, 6, 1, 768, 5, 20, 65, 4, False, True, True),      # own contexts, head size 32
    (192, 12, 1, 192, 5, 3, 20, 3, True, True, True),       # two heads of 16 per CTA
    (64, 4, 1, 128, 5, 6, 50, 140, True, True, True),       # private keys beyond one round of the four parts
    (128, 8, 1, 512, 5, 100, 30, 3, True, True, True),      # eight CTAs, the widest variant within one wave
    (64, 4, 1, 128, 8, 250, 20, 3, False, True, True),      # the widest variant, a context per stream, clusters not full
    (64, 4, 1, 128, 5, 420, 20, 3, False, False, False),    # four CTAs, a context per stream, more streams than one wave
    # one context: the 4-, 8- and 16-row variants of each head size (64: no room for 16 rows), most for models
    # outside the tensor-core chain
    (64, 4, 1, 128, 20, 60, 33, 3, True, True, True),
    (64, 4, 1, 128, 20, 130, 40, 3, True, True, True),
    (64, 4, 2, 128, 20, 199, 65, 3, True, True, True),
    (128, 4, 1, 256, 20, 70, 33, 3, True, True, True),
    (128, 4, 1, 256, 8, 107, 31, 3, True, True, True),
    (128, 4, 1, 256, 5, 201, 64, 3, True, True, True),
    (128, 4, 1, 256, 20, 201, 64, 3, True, False, False),   # no room for the widest variant
    (128, 2, 1, 256, 8, 100, 33, 3, True, True, True),
    (128, 2, 1, 256, 20, 260, 40, 3, True, True, True),
    # where a launch per layer is the faster one
    (128, 4, 1, 256, 5, 200, 4000, 2, True, False, False),
    (64, 2, 2, 128, 5, 3, 6000, 2, True, True, False),
]


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "d%d_h%d_l%d_ff%d_k%d_b%d_nc%d_nt%d_%s" % (*c[:8], "shared" if c[8] else "own"))
def test_sequence_matches_oracle(case, precision):
    import ar_tabpfn
    D, H, L, Dff, K, B, Nc, Nt, shared = case[:9]
    torch.manual_seed(3 + D + Nc)
    m = ar_tabpfn.ARTabPFN(d_model=D, n_heads=H, n_layers=L, d_ff=Dff, num_features=5, num_components=K).eval()
    r = lambda t: t.to(torch.bfloat16).float()
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(r(p))
            p.requires_grad_(False)
    sd = {k: v.clone() for k, v in m.state_dict().items()}
    n = 1 if shared else B
    xs, ys = zip(*[orc.make_dataset(7 * b + 1, Nc + Nt, 5) for b in range(n)])
    x, y = r(torch.stack(xs)).expand(B, -1, -1), r(torch.stack(ys)).expand(B, -1)
    xc, yc, xt = x[:, :Nc], y[:, :Nc], x[:, Nc:]
    # the component of every draw is fixed by a wide margin, so that rounding cannot pick another one
    g = torch.Generator().manual_seed(5)
    expo = torch.rand(Nt, B, K, generator=g) + 0.5
    expo.scatter_(2, torch.randint(K, (Nt, B, 1), generator=g), 1e-5)
    normal = torch.randn(Nt, B, generator=g)
    run = lambda o, f: o.sample_sequence(*(f(t) for t in (xc, yc, xt, expo, normal)), shared=shared)
    want_y, want_ld, want_c = run(orc.OraclePredictor(sd, H), lambda t: t)
    pred = ar_tabpfn.ARTabPFNPredictor.from_trained_model(
        m.cuda(), backend="triton_shared_context" if shared else "flex_attention", precision=precision)
    c = lambda t: t.cuda()
    got_y = pred.sample_sequence(c(xc), c(yc), c(xt), variates=(c(expo), c(normal))).cpu()
    got_ld = pred.last_logdens.cpu()
    assert pred.last_status() == 0
    from ar_tabpfn import _lib
    one_launch = _lib.lib().artab_sequence_workspace(pred._packed(pred._device).ref, ctypes.byref(pred._state)) > 0
    assert one_launch == case[10 if precision == "bf16" else 9]
    assert torch.equal(pred.last_components.cpu(), want_c)
    # Bounds: the bar of the mode plus four times what the mode's arithmetic moves the oracle itself by on
    # this stream (root mean square over its targets): fp32 against fp64; bf16 storage of q / k / v and bf16
    # softmax numerators emulated in the oracle, three realisations.
    if precision == "fp32":
        d = lambda t: t.double()
        alt = [run(orc.OraclePredictor({k: d(v) for k, v in sd.items()}, H), d)]
        bar_y, bar_ld = 1e-5, 3e-5
    else:
        alt = [run(orc.OraclePredictor(sd, H, orc.Emulation(qkv=True, p=True, jitter=j)), lambda t: t) for j in (0, 1, 2)]
        bar_y, bar_ld = 2e-3, 2e-3
    for got, want, k, bar in ((got_y, want_y, 0, bar_y), (got_ld, want_ld, 1, bar_ld)):
        noise = torch.stack([(a[k].double() - want.double()).pow(2).mean(1, keepdim=True) for a in alt]).mean(0).sqrt()
        err = (got.double() - want.double()).abs()
        bound = bar * (1 + want.double().abs()) + 4 * noise
        assert bool((err <= bound).all()), (k, float(err.max()), float((err / bound).max()))


def test_workspace_is_given_back_and_a_job_that_has_no_room_for_it_still_runs(monkeypatch):
    import ar_tabpfn
    torch.manual_seed(4)
    m = ar_tabpfn.ARTabPFN(num_features=5).eval().cuda()
    pred = ar_tabpfn.ARTabPFNPredictor.from_trained_model(m, backend="triton_shared_context", precision="fp32")
    B, Nc, Nt, K = 9, 2000, 5, 5
    g = torch.Generator(device="cuda").manual_seed(1)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    expo = torch.rand(Nt, B, K, device="cuda", generator=g) + 0.5
    expo.scatter_(2, torch.randint(K, (Nt, B, 1), device="cuda", generator=g), 1e-5)
    args = r(1, Nc, 5).expand(B, -1, -1), r(1, Nc).expand(B, -1), r(1, Nt, 5).expand(B, -1, -1)
    run = lambda: pred.sample_sequence(*args, variates=(expo, normal))
    normal = r(Nt, B)
    asked = []
    plain = type(pred)._sequence_workspace
    monkeypatch.setattr(type(pred), "_sequence_workspace", lambda self, need: asked.append(need) or plain(self, need))
    want = run().clone()
    assert asked[-1] > 1 << 20
    held = torch.cuda.memory_allocated()
    run()
    assert torch.cuda.memory_allocated() <= held and not any(t.dtype == torch.uint8 for t in pred._bufs.values())
    monkeypatch.undo()

    def no_room(n, *a, dtype=None, **k):
        if dtype is torch.uint8:
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(n, *a, dtype=dtype, **k)
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", no_room)
    got = run()
    torch.testing.assert_close(got, want, atol=1e-4, rtol=1e-4)   # fp32 sums in another order, five targets deep
