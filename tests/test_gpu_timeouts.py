"""The give-up path of the bounded device-side waits, exercised without faulting anything: a
diagnostic switch makes the context contraction's MMA thread withhold its "scores ready" signal and
the wait limit is set to a fraction of a millisecond, so the softmax threads' waits run out, the
CTAs write nothing, free what they hold and the kernel returns normally with a non-zero status."""
import pytest
import torch

from util import ref_attention

pytestmark = pytest.mark.gpu


def _problem(rows=96, H=2, Nc=100, Dh=32):
    from ar_tabpfn.model import triton_kernels as tk
    g = torch.Generator(device="cuda").manual_seed(5)
    q = torch.randn(rows, H, Dh, device="cuda", generator=g).bfloat16()
    k = torch.randn(H, Nc, Dh, device="cuda", generator=g).bfloat16()
    v = torch.randn(H, Nc, Dh, device="cuda", generator=g).bfloat16()
    kp, vp, _, Ncp = tk.pack_context(k, v)
    return q, k, v, kp, vp, Ncp


def _ctx(lib, _lib, q, kp, vp, Nc, Ncp, out, lse, status, splits=1):
    rows, H, Dh = q.shape
    return lib.artab_context_attention(_lib.BF16, _lib.ptr(q), _lib.ptr(kp), _lib.ptr(vp), rows, rows, 1, H, Dh, Nc,
                                       Ncp, splits, _lib.ptr(out), _lib.ptr(lse), _lib.ptr(status),
                                       _lib.stream_ptr())


def test_wait_runs_out_status_is_set_and_the_next_launch_is_correct():
    from ar_tabpfn import _lib
    lib = _lib.lib()
    q, k, v, kp, vp, Ncp = _problem()
    rows, H, Dh = q.shape
    Nc = k.shape[1]
    out = torch.full((1, rows, H, Dh), -7.0, device="cuda")
    lse = torch.full((1, rows, H), -7.0, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    try:
        _lib.check(lib.artab_debug_set(_lib.DEBUG_WAIT_CYCLES, 200_000))       # ~0.1 ms
        _lib.check(lib.artab_debug_set(_lib.DEBUG_DROP_SCORE_COMMITS, 1))
        rc = _ctx(lib, _lib, q, kp, vp, Nc, Ncp, out, lse, status)
        torch.cuda.synchronize()
    finally:
        lib.artab_debug_set(_lib.DEBUG_DROP_SCORE_COMMITS, 0)
        lib.artab_debug_set(_lib.DEBUG_WAIT_CYCLES, 0)
    assert rc == 0                                   # the launch itself succeeded ...
    assert int(status.item()) != 0                   # ... the kernel reports that a wait gave up ...
    assert bool((out == -7.0).all()) and bool((lse == -7.0).all())   # ... and wrote no result
    # the context is intact: the same call without the switch is correct
    status.zero_()
    _lib.check(_ctx(lib, _lib, q, kp, vp, Nc, Ncp, out, lse, status))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    want, want_lse = ref_attention(q.permute(1, 0, 2).unsqueeze(0), k.unsqueeze(0), v.unsqueeze(0))
    got = out[0].permute(1, 0, 2).unsqueeze(0)
    assert float((got - want).abs().max() / want.abs().max()) <= 1e-2
    torch.testing.assert_close(lse[0].t().unsqueeze(0), want_lse, atol=2e-3, rtol=0)


def test_noalloc_entry_reports_a_timed_out_wait_as_nan():
    from ar_tabpfn import _lib
    lib = _lib.lib()
    q, k, v, kp, vp, Ncp = _problem(rows=64, Nc=300)
    rows, H, Dh = q.shape
    Nc = k.shape[1]
    out = torch.zeros(rows, H, Dh, device="cuda")

    def call():
        return lib.artab_context_attention_noalloc(_lib.BF16, _lib.ptr(q), _lib.ptr(kp), _lib.ptr(vp), rows, rows, 1,
                                                   H, Dh, Nc, Ncp, 2, _lib.ptr(out), _lib.stream_ptr())
    _lib.check(call())       # also the one-off look-up of the built-in array, outside the failing call
    torch.cuda.synchronize()
    good = out.clone()
    try:
        _lib.check(lib.artab_debug_set(_lib.DEBUG_WAIT_CYCLES, 200_000))
        _lib.check(lib.artab_debug_set(_lib.DEBUG_DROP_SCORE_COMMITS, 1))
        rc = call()
        torch.cuda.synchronize()
    finally:
        lib.artab_debug_set(_lib.DEBUG_DROP_SCORE_COMMITS, 0)
        lib.artab_debug_set(_lib.DEBUG_WAIT_CYCLES, 0)
    assert rc == 0 and bool(torch.isnan(out).all())   # never a plausible mix of stale partials
    _lib.check(call())
    torch.cuda.synchronize()
    assert torch.equal(out, good)


def test_hybrid_attention_timed_out_call_is_nan_and_the_next_one_is_not():
    from ar_tabpfn import _lib
    from ar_tabpfn.model import triton_kernels as tk
    lib = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    args = r(70, 2, 1, 32), r(2, 300, 32), r(2, 300, 32), r(70, 2, 9, 32), r(70, 2, 9, 32)
    good = tk.hybrid_attention(*args)
    assert int(tk.last_status.item()) == 0
    try:
        _lib.check(lib.artab_debug_set(_lib.DEBUG_WAIT_CYCLES, 200_000))
        _lib.check(lib.artab_debug_set(_lib.DEBUG_DROP_SCORE_COMMITS, 1))
        bad = tk.hybrid_attention(*args)
        torch.cuda.synchronize()
    finally:
        lib.artab_debug_set(_lib.DEBUG_DROP_SCORE_COMMITS, 0)
        lib.artab_debug_set(_lib.DEBUG_WAIT_CYCLES, 0)
    word = tk.last_status
    assert int(word.item()) != 0 and bool(torch.isnan(bad).all())
    assert torch.equal(tk.hybrid_attention(*args), good)      # every call has a word of its own ...
    assert int(tk.last_status.item()) == 0 and int(word.item()) != 0
    # ... written by the call itself, whatever its memory held before
    q, k, v, kb, vb = args
    out, ws = torch.empty_like(q), torch.empty(1 << 20, dtype=torch.uint8, device="cuda")
    _lib.check(lib.artab_hybrid_attention(_lib.BF16, *(_lib.ptr(t) for t in args), None, None, 70, 2, 1, 32, 300, 9,
                                          _lib.ptr(out), _lib.ptr(ws), ws.numel(), _lib.ptr(word), _lib.stream_ptr()))
    assert torch.equal(out, good) and int(word.item()) == 0


def test_predictor_raises_after_a_timed_out_call():
    from ar_tabpfn import _lib
    from ar_tabpfn.model import ARTabPFNPredictor
    import synthetic as syn
    lib = _lib.lib()
    m = syn.build_model(6, 9, d_model=64, n_heads=2, n_layers=2, d_ff=256).cuda()
    p = ARTabPFNPredictor.from_trained_model(m, backend="triton_shared_context", precision="bf16")
    g = torch.Generator(device="cuda").manual_seed(1)
    xc, yc = torch.randn(4, 40, 6, device="cuda", generator=g), torch.randn(4, 40, device="cuda", generator=g)
    xt, yt = torch.randn(4, 5, 6, device="cuda", generator=g), torch.randn(4, 5, device="cuda", generator=g)
    good = p.evaluate_joint_density(xc, yc, xt, yt).clone()
    assert p.last_status() == 0
    try:
        _lib.check(lib.artab_debug_set(_lib.DEBUG_WAIT_CYCLES, 200_000))
        _lib.check(lib.artab_debug_set(_lib.DEBUG_DROP_SCORE_COMMITS, 1))
        p.evaluate_joint_density(xc, yc, xt, yt)
        torch.cuda.synchronize()
    finally:
        lib.artab_debug_set(_lib.DEBUG_DROP_SCORE_COMMITS, 0)
        lib.artab_debug_set(_lib.DEBUG_WAIT_CYCLES, 0)
    assert p.last_status() != 0
    with pytest.raises(_lib.ArtabError, match="wait gave up"):
        p.evaluate_joint_density(xc, yc, xt, yt)
    # the error is reported once; the predictor then works again
    assert torch.equal(p.evaluate_joint_density(xc, yc, xt, yt), good)
    assert p.last_status() == 0


def _network(precision, **cfg):
    from ar_tabpfn import ARTabPFN
    from ar_tabpfn.model import ARTabPFNPredictor
    torch.manual_seed(2)
    m = ARTabPFN(num_features=4, num_components=5, **cfg).eval()
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(p.bfloat16().float())
    return ARTabPFNPredictor.from_trained_model(m.cuda(), backend="triton_shared_context", precision=precision)


def _rows(B, Nc, Nt):
    g = torch.Generator(device="cuda").manual_seed(6)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    return r(1, Nc, 4).expand(B, -1, -1), r(1, Nc).expand(B, -1), r(B, Nt, 4), r(B, Nt)


@pytest.mark.parametrize("precision,code,cfg", [
    # head size 16: the contraction and the private pass have no bounded waits, the dense chain is the only one
    ("bf16", 6, dict(d_model=64, n_heads=4, n_layers=1, d_ff=128)),
    ("bf16", 6, dict(d_model=64, n_heads=4, n_layers=3, d_ff=256)),
    ("bf16", 6, dict(d_model=192, n_heads=12, n_layers=2, d_ff=384)),
    ("fp32", 5, dict(d_model=64, n_heads=4, n_layers=1, d_ff=128)),
    ("fp32", 5, dict(d_model=128, n_heads=4, n_layers=2, d_ff=256)),
    ("fp32", 5, dict(d_model=192, n_heads=6, n_layers=2, d_ff=768)),
])
def test_dense_chain_gives_up_and_the_next_call_is_correct(precision, code, cfg):
    """The few-row (6) and the register-tiled chain (5), with a limit of one cycle."""
    from ar_tabpfn import _lib
    lib = _lib.lib()
    p = _network(precision, **cfg)
    args = _rows(5, 70, 9)
    good = p.evaluate_joint_density(*args).clone()
    assert p.last_status() == 0 and bool(good.isfinite().all())
    try:
        _lib.check(lib.artab_debug_set(_lib.DEBUG_WAIT_CYCLES, 1))
        p.evaluate_joint_density(*args)
        torch.cuda.synchronize()
    finally:
        lib.artab_debug_set(_lib.DEBUG_WAIT_CYCLES, 0)
    assert p.last_status() == code
    with pytest.raises(_lib.ArtabError, match="wait gave up"):
        p.evaluate_joint_density(*args)
    assert torch.equal(p.evaluate_joint_density(*args), good)
    assert p.last_status() == 0


@pytest.mark.parametrize("B,heads,Nc", [(1, 4, 40), (130, 4, 1100), (40, 8, 33), (9, 12, 70)])
def test_whole_sequence_decode_gives_up_and_the_next_one_is_correct(B, heads, Nc):
    """A limit of one cycle: the first wait for a copy or a peer that has not arrived yet ends the job in every CTA."""
    import ctypes as C
    from ar_tabpfn import _lib
    lib = _lib.lib()
    p = _network("fp32", d_model=192 if heads == 12 else 128, n_heads=heads, n_layers=3, d_ff=384 if heads == 12 else 256)
    Nt = 7
    xc, yc, xt, _ = _rows(B, Nc, Nt)
    expo, normal = torch.rand(Nt, B, 5, device="cuda") + 0.1, torch.randn(Nt, B, device="cuda")
    p.init_kv_cache(B, Nt, xc.device, torch.float32)
    p.prefill_context(xc, yc)
    pm, st = p._packed(p._device), p._state
    need = int(lib.artab_sequence_workspace(pm.ref, C.byref(st)))
    assert need > 0
    pm.prepare_sequence()
    ws, status = torch.empty(need, dtype=torch.uint8, device="cuda"), p._bufs["status"]

    def decode():
        samples, ld = torch.full((B, Nt), -7.0, device="cuda"), torch.empty(B, Nt, device="cuda")
        comp = torch.empty(B, Nt, dtype=torch.int32, device="cuda")
        st.buffer_len = 0
        status.zero_()
        _lib.check(lib.artab_decode_sequence(pm.ref, C.byref(st), _lib.ptr(xt), Nt * 4, 4, Nt, 0, Nt, _lib.ptr(samples),
                                             _lib.ptr(expo), _lib.ptr(normal), _lib.ptr(ld), _lib.ptr(comp), _lib.ptr(ws),
                                             need, _lib.stream_ptr()))
        torch.cuda.synchronize()
        return samples, int(status.item())
    good, code = decode()
    assert code == 0 and bool(good.isfinite().all()) and bool((good != -7.0).all())
    try:
        _lib.check(lib.artab_debug_set(_lib.DEBUG_WAIT_CYCLES, 1))
        void, code = decode()
    finally:
        lib.artab_debug_set(_lib.DEBUG_WAIT_CYCLES, 0)
    assert code == 4 and not bool(void.any())
    again, code = decode()
    assert code == 0 and torch.equal(again, good)


@pytest.mark.parametrize("precision,d_ff", [("fp32", 256), ("bf16", 128)])
def test_results_of_a_sampling_call_that_gave_up_are_zero(precision, d_ff):
    """Not what an earlier call left in the same memory."""
    from ar_tabpfn import _lib
    lib = _lib.lib()
    p = _network(precision, d_model=64, n_heads=4, n_layers=2, d_ff=d_ff)
    B, Nt = 6, 11
    xc, yc, xt, _ = _rows(B, 50, Nt)
    variates = torch.rand(Nt, B, 5, device="cuda") + 0.1, torch.randn(Nt, B, device="cuda")
    p.sample_sequence(xc, yc, xt, variates=variates)
    torch.cuda.synchronize()
    try:
        _lib.check(lib.artab_debug_set(_lib.DEBUG_WAIT_CYCLES, 1))
        void = p.sample_sequence(xc, yc, xt, variates=variates)
        torch.cuda.synchronize()
    finally:
        lib.artab_debug_set(_lib.DEBUG_WAIT_CYCLES, 0)
    assert p.last_status() != 0
    assert not bool(void.any()) and not bool(p.last_logdens.any()) and not bool(p.last_components.any())
