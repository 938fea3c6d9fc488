"""Passes whose contractions claim their work items against the same passes with the items dealt out: bit for bit, and again when
a contraction is launched once more without the kernel that zeroes the words the items are claimed from."""
import pytest
import torch

from moe_explore import _native
from moe_explore.expert_compute import routed_expert_compute
from moe_explore.triton_kernels.m_grouped_gemm import MGroupedGEMMParams, m_grouped_gemm

pytestmark = pytest.mark.gpu

ONCE = {"moe_expert_forward": _native.FWD_ROUTE | _native.FWD_DISPATCH, "moe_expert_backward": _native.BWD_FOLD,
        "moe_rows_gemm": _native.ROWS_LAYOUT}


@pytest.fixture
def launch(monkeypatch):
    real, how = _native.run_pass, {}

    def run_pass(name, p, steps, rows):
        if how["mode"] == "dealt out":
            p.counters = None
        real(name, p, steps, rows)
        if how["mode"] == "twice":
            real(name, p, [s for s in steps if not s[0] & ONCE[name]], rows)
    monkeypatch.setattr(_native, "run_pass", run_pass)
    return lambda mode: how.update(mode=mode)


@pytest.mark.parametrize("act,dtype", [("swiglu", torch.bfloat16), ("gelu", torch.float16)])
@pytest.mark.parametrize("T,E,spread", [(2000, 96, 1.0), (700, 128, 3.0), (9000, 96, 0.0)])   # some experts without a row at 3.0
def test_claimed_and_dealt_out_items(T, E, spread, act, dtype, launch, native):
    d, inter, k = 520, 1032, 4
    g = torch.Generator(device="cuda").manual_seed(T)
    mk = lambda *s, std=1.0: (torch.randn(*s, generator=g, device="cuda") * std).to(dtype)
    ids = torch.topk(torch.randn(T, E, generator=g, device="cuda") + spread * torch.randn(E, generator=g, device="cuda"), k).indices
    leaves = [mk(T, d), torch.rand(T, k, generator=g, device="cuda").to(dtype), mk(E, d, 2 * inter if act == "swiglu" else inter, std=0.1),
              mk(E, inter, d, std=0.1)]
    grad = mk(T, d)

    def run(mode):
        launch(mode)
        p = [t.clone().requires_grad_() for t in leaves]
        out = routed_expert_compute(*p, ids, E, k, act)
        got = [out.detach(), *torch.autograd.grad(out, p, grad)]
        with torch.no_grad():
            got.append(routed_expert_compute(*p, ids, E, k, act))
        groups = torch.bincount(ids.flatten(), minlength=E).cumsum(0).int()
        groups = torch.cat([groups.new_zeros(1), groups])
        got.append(m_grouped_gemm(mk(T * k, d) * 0 + 1, MGroupedGEMMParams(leaves[2], groups, None, False, False, T * k, 1)))
        return got

    ref = run("dealt out")
    for mode in ("claimed", "claimed", "twice"):
        assert all(torch.equal(a, b) for a, b in zip(run(mode), ref)), mode


def test_nothing_to_claim(launch, native):
    """Every id out of range: no row tile is in use, the words stay as they are."""
    from moe_explore.routing_plan import device_status

    T, E, d, inter = 3000, 96, 136, 1032
    x, w1, w2 = (torch.randn(*s, device="cuda").bfloat16() for s in ((T, d), (E, d, 2 * inter), (E, inter, d)))
    scores, ids = torch.ones(T, 2, device="cuda").bfloat16(), torch.full((T, 2), E, device="cuda")
    launch("twice")
    p = [t.requires_grad_() for t in (x, scores, w1, w2)]
    out = routed_expert_compute(*p, ids, E, 2, "swiglu")
    assert all(not t.any() for t in (out, *torch.autograd.grad(out, p, torch.ones_like(out))))
    assert native.read_status(device_status(), reset=True) == 100
