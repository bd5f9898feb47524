"""Shapes handed to hybrid_attention, checked before anything reaches the device: the native entry point sees
addresses only, so an extent that does not fit must be refused (or routed to the general form) in Python."""
import pytest
import torch

from ar_tabpfn import _lib
from ar_tabpfn.model import triton_kernels as tk

B, H, Dh, Nc, Nb = 3, 2, 16, 9, 5


class FakeLibrary:
    """Records the native calls instead of making them."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append((name, args))
            return 64 if name.endswith("workspace") else 1 if name == "artab_plan_splits" else 0
        return call

    def names(self):
        return [n for n, _ in self.calls]


@pytest.fixture
def fake(monkeypatch):
    lib = FakeLibrary()
    monkeypatch.setattr(_lib, "lib", lambda: lib)
    monkeypatch.setattr(_lib, "stream_ptr", lambda: None)
    return lib


def _args(**shapes):
    s = dict(q=(B, H, 1, Dh), k_ctx=(H, Nc, Dh), v_ctx=(H, Nc, Dh), k_buf=(B, H, Nb, Dh), v_buf=(B, H, Nb, Dh))
    s.update(shapes)
    return [torch.zeros(s[n]) for n in ("q", "k_ctx", "v_ctx", "k_buf", "v_buf")]


@pytest.mark.parametrize("shapes", [
    dict(v_buf=(B, H, Nb - 1, Dh)), dict(v_buf=(1, H, Nb, Dh)), dict(k_buf=(1, H, Nb, Dh), v_buf=(1, H, Nb, Dh)),
    dict(k_buf=(B, 1, Nb, Dh), v_buf=(B, 1, Nb, Dh)), dict(v_ctx=(H, Nc - 1, Dh)), dict(v_ctx=(H, Nc, Dh // 2)),
    dict(k_ctx=(1, Nc, Dh), v_ctx=(1, Nc, Dh)), dict(k_ctx=(H, Nc, 32), v_ctx=(H, Nc, 32)),
    dict(k_ctx=(B, 1, Nc, Dh), v_ctx=(B, 1, Nc, Dh)), dict(k_ctx=(Nc, Dh), v_ctx=(Nc, Dh)),
], ids=str)
def test_shapes_that_do_not_fit_raise_before_any_launch(fake, shapes):
    with pytest.raises((ValueError, RuntimeError)):
        tk.hybrid_attention(*_args(**shapes))
    assert not [n for n in fake.names() if "attention" in n]


@pytest.mark.parametrize("shapes,groups", [(dict(k_ctx=(B, H, Nc, Dh), v_ctx=(B, H, Nc, Dh)), B),
                                           (dict(v_ctx=(1, Nc, Dh)), 1), (dict(v_ctx=(1, H, Nc, Dh)), 1)], ids=str)
def test_other_accepted_shapes_take_the_general_form(fake, shapes, groups):
    tk.hybrid_attention(*_args(**shapes))
    args = dict(fake.calls)["artab_context_attention"]
    assert "artab_hybrid_attention" not in fake.names()
    assert args[6] == groups and args[9] == Nc           # n_groups, n_ctx


def test_plain_shapes_take_the_two_launch_form(fake):
    for lead in ((), (1,)):
        fake.calls.clear()
        tk.hybrid_attention(*_args(k_ctx=(*lead, H, Nc, Dh), v_ctx=(*lead, H, Nc, Dh)))
        assert fake.names() == ["artab_hybrid_workspace", "artab_hybrid_attention"]
        assert fake.calls[1][1][12] == Nc


@pytest.mark.parametrize("Lq", [1, 3])
def test_unaligned_queries_are_copied_to_an_aligned_address(fake, Lq):
    a = _args()
    a[0] = torch.zeros(1 + B * Lq * Dh)[1:].view(B, 1, Lq, Dh)      # one head: the token-major view starts here too
    a[1:] = [t[..., :1, :, :].contiguous() for t in a[1:]]
    tk.hybrid_attention(*a)
    assert fake.calls[1][1][1] % 16 == 0
