"""bf16 mode at the row counts and sizes where the few-row chain changes what it does: one row, a whole 32-row
cluster and one row more, the last row count of one wave of clusters and the first beyond it (tcgen05 chain); one to
eight 32-wide hidden slices per CTA; weights with and without a low part."""
import pytest
import torch

import artab_oracle as orc

pytestmark = pytest.mark.gpu

CASES = [
    # d_model, heads, d_ff, components, streams, context rows, targets, weights exact in bf16
    (192, 6, 768, 5, 1, 33, 1, True),      # two target rows; context one row past a cluster
    (192, 6, 1024, 5, 4, 32, 4, False),    # one whole cluster; eight hidden slices, two column pairs per warp
    (192, 3, 128, 5, 31, 31, 1, True),     # head size 64; one hidden slice
    (128, 4, 256, 5, 24, 1185, 23, True),  # context beyond one wave; 1104 target rows
    (128, 8, 640, 2, 5, 97, 7, False),     # head size 16; odd number of hidden slices
    (64, 2, 128, 5, 64, 10, 18, True),     # 2304 target rows: beyond one wave
    (64, 1, 512, 5, 3, 65, 9, False),      # one head
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "d%d_h%d_ff%d_k%d_b%d_nc%d_nt%d_exact%d" % c)
def test_bf16_joint_density_at_row_edges(case):
    import ar_tabpfn
    D, H, Dff, K, B, Nc, Nt, exact = case
    torch.manual_seed(D + Nc)
    m = ar_tabpfn.ARTabPFN(d_model=D, n_heads=H, n_layers=2, d_ff=Dff, num_features=4, num_components=K).eval()
    for p in m.parameters():
        p.requires_grad_(False)
        if exact:
            p.copy_(p.to(torch.bfloat16).float())
    sd = {k: v.clone() for k, v in m.state_dict().items()}
    g = torch.Generator().manual_seed(1)
    r = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16).float()
    x, y = r(1, Nc + Nt, 4).expand(B, -1, -1), r(B, Nc + Nt)
    y[:, :Nc] = y[:1, :Nc]
    args = (x[:, :Nc], y[:, :Nc], x[:, Nc:], y[:, Nc:])
    want = orc.OraclePredictor(sd, H).evaluate_joint_density(*args)
    # what rounding q, k, v and the softmax numerators to bf16 costs the oracle on each target (root mean square over
    # five realisations); four times that, above the 2e-3 bar of the mode
    devs = [orc.OraclePredictor(sd, H, orc.Emulation(qkv=True, p=True, jitter=s)).evaluate_joint_density(*args) - want
            for s in range(5)]
    bound = 2e-3 + 4 * torch.stack(devs).pow(2).mean(0).sqrt()
    pred = ar_tabpfn.ARTabPFNPredictor.from_trained_model(m.cuda(), backend="triton_shared_context", precision="bf16")
    got = pred.evaluate_joint_density(*(t.cuda() for t in args)).cpu()
    assert pred.last_status() == 0
    err = (got - want).abs()
    assert bool((err <= bound).all()), (float(err.max()), float((err / bound).max()))
    # one sample path per stream: the density of what was drawn agrees with teacher forcing up to the same rounding
    with torch.no_grad():
        pred.ar_tokens.zero_()   # sampling and teacher forcing number the AR tokens differently
    ys = pred.sample_sequence(*(t.cuda() for t in args[:3]))
    ld = pred.last_logdens.clone()
    gap = (pred.evaluate_joint_density(*(t.cuda() for t in args[:3]), ys) - ld).abs()
    assert bool(torch.isfinite(ys).all()) and float(gap.median()) <= 2e-3


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_layouts_in_turn_on_one_predictor(precision):
    """Context lengths with and without padding of the key axis, in turn on one predictor whose buffers are reused:
    the same bits as a predictor of its own gives."""
    import ar_tabpfn
    torch.manual_seed(3)
    m = ar_tabpfn.ARTabPFN(d_model=64, n_heads=2, n_layers=2, d_ff=128, num_features=4).eval().cuda()
    make = lambda: ar_tabpfn.ARTabPFNPredictor.from_trained_model(m, backend="flex_attention", precision=precision)
    kept, other = make(), make()
    for Nc, B, Nt in ((50, 3, 6), (43, 3, 6), (43, 3, 6), (50, 3, 6), (50, 2, 9), (48, 3, 6)):
        g = torch.Generator(device="cuda").manual_seed(Nc + B)
        x, y = torch.randn(B, Nc + Nt, 4, generator=g, device="cuda"), torch.randn(B, Nc + Nt, generator=g, device="cuda")
        args = (x[:, :Nc], y[:, :Nc], x[:, Nc:], y[:, Nc:])
        got = kept.evaluate_joint_density(*args)
        assert m.backbone.layers[1].k_ctx_cache.shape[2] == Nc
        other.evaluate_joint_density(*args)   # takes the modules' cache views for itself
        assert torch.equal(got, make().evaluate_joint_density(*args))
