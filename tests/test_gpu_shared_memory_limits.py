"""A kernel's shared-memory limit is one attribute per device: neither an occupancy query nor a smaller job, on
whatever host thread, may lower it below what a launch relies on."""
import ctypes as C
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _on_a_thread(f):
    """On a fresh host thread (the occupancy figures are kept per thread); errors are raised here."""
    out = []

    def body():
        try:
            out.append((f(), None))
        except BaseException as e:  # noqa: BLE001  (handed to the caller)
            out.append((None, e))
    t = threading.Thread(target=body)
    t.start()
    t.join()
    if out[0][1] is not None:
        raise out[0][1]
    return out[0][0]


def _predictor(precision, **cfg):
    import ar_tabpfn
    torch.manual_seed(1)
    m = ar_tabpfn.ARTabPFN(num_features=3, num_components=5, n_layers=1, **cfg).eval()
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(p.bfloat16().float())
    return ar_tabpfn.ARTabPFNPredictor.from_trained_model(m.cuda(), backend="triton_shared_context", precision=precision)


def _sample(pred, B=8, Nc=20, Nt=3):
    g = torch.Generator(device="cuda").manual_seed(2)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, y, xt = r(1, Nc, 3).expand(B, -1, -1), r(1, Nc).expand(B, -1), r(1, Nt, 3).expand(B, -1, -1)
    expo = torch.empty(Nt, B, 5, device="cuda").exponential_(generator=g)
    return pred.sample_sequence(x, y, xt, variates=(expo, r(Nt, B))).clone()


def test_few_row_chain_of_several_hidden_widths_on_two_threads():
    small, middle, large = (_predictor("bf16", d_model=64, n_heads=2, d_ff=f) for f in (256, 512, 1024))

    def density(p, B=8):
        g = torch.Generator(device="cuda").manual_seed(3)
        r = lambda *s: torch.randn(*s, device="cuda", generator=g)
        return p.evaluate_joint_density(r(B, 20, 3), r(B, 20), r(B, 4, 3), r(B, 4)).clone()
    density(small)
    want = density(large)
    _on_a_thread(lambda: density(middle))
    assert torch.equal(density(large), want)
    torch.cuda.synchronize()


def test_whole_sequence_path_after_a_smaller_job_of_the_queried_variant():
    from ar_tabpfn import _lib
    lib = _lib.lib()
    four, eight = _predictor("fp32", d_model=128, n_heads=4, d_ff=256), _predictor("fp32", d_model=128, n_heads=8, d_ff=256)
    _on_a_thread(lambda: _sample(four, B=130))       # four streams per cluster: the variant the queries use

    def applies():
        _sample(eight)
        return int(lib.artab_sequence_workspace(eight._packed(eight._device).ref, C.byref(eight._state)))
    assert _on_a_thread(applies) > 0


def test_a_refused_launch_does_not_surface_in_the_callers_next_operation():
    """More heads than a grid has rows: the launch is refused on the host, nothing runs."""
    from ar_tabpfn import _lib
    lib = _lib.lib()
    b = torch.zeros(64, dtype=torch.bfloat16, device="cuda")
    f = torch.zeros(64, device="cuda")
    with pytest.raises(_lib.ArtabError):
        _lib.check(lib.artab_context_attention(_lib.BF16, _lib.ptr(b), _lib.ptr(b), _lib.ptr(b), 1, 1, 1, 70000, 32, 8, 8, 1,
                                               _lib.ptr(f), _lib.ptr(f), None, _lib.stream_ptr()))
    assert float((f + 1).sum()) == 64.0
