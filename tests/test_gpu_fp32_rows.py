"""fp32 mode at the row counts where the register-tiled kernels change their tile: 1, 2, 4 and 8 rows per thread
of the dense chain (by rows), 2, 4 and 8 query rows per warp of the context attention (by rows of a group), head
sizes 16, 32 and 64, context tiles of 32 and stages of 64 keys with remainders."""
import pytest
import torch

import artab_oracle as orc

pytestmark = pytest.mark.gpu

# d_model, heads, d_ff, components, datasets, context rows, targets
CASES = [
    (64, 4, 128, 20, 60, 79, 3),      # 4740 context rows: two rows per thread; head size 16
    (64, 2, 192, 5, 500, 19, 2),      # 9500: four; three hidden chunks
    (64, 1, 64, 5, 2112, 9, 1),       # 19008: eight; groups of nine rows, head size 64
    (128, 4, 256, 5, 17, 70, 4),      # 1190: two; stage of 64 keys and six more
    (128, 8, 128, 5, 74, 32, 2),      # 2368: two, all row groups full; head size 16
    (128, 2, 384, 8, 65, 73, 2),      # 4745: eight; head size 64
    (192, 6, 192, 5, 37, 65, 2),      # 2405: four
    (192, 3, 768, 5, 150, 33, 1),     # 4950: eight; head size 64, four hidden chunks
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "d%d_h%d_ff%d_k%d_b%d_nc%d_nt%d" % c)
def test_fp32_joint_density_at_tile_edges(case):
    import ar_tabpfn
    D, H, Dff, K, B, Nc, Nt = case
    torch.manual_seed(D + Nc)
    m = ar_tabpfn.ARTabPFN(d_model=D, n_heads=H, n_layers=2, d_ff=Dff, num_features=4, num_components=K).eval()
    for p in m.parameters():
        p.requires_grad_(False)
    sd = {k: v.clone() for k, v in m.state_dict().items()}
    g = torch.Generator().manual_seed(1)
    x, y = torch.randn(B, Nc + Nt, 4, generator=g), torch.randn(B, Nc + Nt, generator=g)
    args = (x[:, :Nc], y[:, :Nc], x[:, Nc:], y[:, Nc:])
    want = orc.OraclePredictor(sd, H).evaluate_joint_density(*args, shared=False)
    d = lambda t: t.double()
    want64 = orc.OraclePredictor({k: d(v) for k, v in sd.items()}, H).evaluate_joint_density(*map(d, args), shared=False)
    pred = ar_tabpfn.ARTabPFNPredictor.from_trained_model(m.cuda(), backend="flex_attention", precision="fp32")
    got = pred.evaluate_joint_density(*(t.cuda() for t in args)).cpu()
    assert pred.last_status() == 0
    # The fp32 bar plus four times the oracle's own fp32-against-fp64 difference (root mean square over the
    # call).  With twenty narrow components a target can sit 20 standard deviations out (log density -279): its
    # -z^2 / 2 carries twice the relative error of (y - mean) / std, so the bar is relative there.
    noise = float((want.double() - want64).pow(2).mean().sqrt())
    err = (got - want).abs()
    assert bool((err <= 1e-5 * (1 + want.abs()) + 4 * noise).all()), (float(err.max()), noise)


# dtype, head size, keys, pitch of the key axis, elements K / V / out start after a 16-byte boundary
PLACES = [
    (torch.bfloat16, 16, 50, 50, 0),    # transposed V with a pitch of no whole float4s
    (torch.bfloat16, 64, 70, 71, 0),    # odd pitch
    (torch.bfloat16, 16, 33, 40, 3),    # whole pitch, arrays off the boundary
    (torch.float32, 32, 65, 65, 1),
    (torch.float32, 64, 40, 41, 2),
]


@pytest.mark.parametrize("place", PLACES, ids=lambda p: "%s_dh%d_nc%d_pitch%d_off%d" % (str(p[0])[6:], *p[1:]))
def test_context_attention_takes_any_placement(place):
    import ar_tabpfn  # noqa: F401
    from ar_tabpfn import _lib
    dtype, Dh, Nc, Ncp, off = place
    H, rows = 2, 11
    g = torch.Generator().manual_seed(Nc)
    q, k, v = (torch.randn(n, H, Dh, generator=g).to(dtype) for n in (rows, Nc, Nc))
    kp = torch.zeros(H, Ncp, Dh, dtype=dtype)
    kp[:, :Nc] = k.transpose(0, 1)
    if dtype == torch.bfloat16:
        vp = torch.zeros(H, 2 * Dh, Ncp, dtype=dtype)
        vp[:, :Dh, :Nc] = v.permute(1, 2, 0)
    else:
        vp = torch.zeros(H, Ncp, Dh, dtype=dtype)
        vp[:, :Nc] = v.transpose(0, 1)

    def placed(t):
        buf = torch.zeros(t.numel() + off + 8, dtype=t.dtype, device="cuda")
        at = buf[off:off + t.numel()]
        at.copy_(t.reshape(-1))
        return at

    kd, vd, out = placed(kp), placed(vp), placed(torch.zeros(rows, H, Dh))
    qd, lse = q.cuda(), torch.empty(rows, H, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.check(_lib.lib().artab_context_attention(_lib.dtype_code(dtype), _lib.ptr(qd), _lib.ptr(kd), _lib.ptr(vd), rows,
                                                  rows, 1, H, Dh, Nc, Ncp, 1, _lib.ptr(out), _lib.ptr(lse),
                                                  _lib.ptr(status), _lib.stream_ptr()))
    s = torch.einsum("rhd,khd->rhk", q.double(), k.double()) / Dh ** 0.5
    want = torch.einsum("rhk,khd->rhd", s.softmax(-1), v.double())
    # fp32 arithmetic on the stored values: sums over at most 70 keys
    torch.testing.assert_close(out.view(rows, H, Dh).cpu().double(), want, atol=1e-5, rtol=1e-5)
    torch.testing.assert_close(lse.cpu().double(), s.logsumexp(-1), atol=1e-5, rtol=1e-5)
