"""Router and choice in one launch, and the experts' order by rounds of a warp: sizes around a CTA's tokens and a warp's round, ties, NaN and
infinities, ids of no expert."""
import pytest
import torch

from dgi_b200 import mixer_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,E,top,width", [(1, 8, 2, 1024), (7, 3, 3, 30), (2368, 8, 2, 512), (2500, 5, 1, 516), (4099, 8, 4, 1024), (2400, 1, 1, 64), (9, 12, 2, 64)])
def test_router_and_choice(n, E, top, width, dtype):
    """The same ids and weights to the bit as the two launches, whose logits are the same sums."""
    gen = torch.Generator(device="cuda").manual_seed(n + E)
    x = torch.randn(n, width, generator=gen, device="cuda").to(dtype)
    w = torch.randn(E, width, generator=gen, device="cuda") / width ** 0.5
    if E > 2:
        w[2] = w[0]                                  # ties
    x[n // 2, 3] = float("nan")                      # a token of NaNs
    x[n - 1] = 0.0                                   # all logits alike
    ids, weights = mixer_ops.router_sigmoid_topk(x, w, top)
    want, want_w = mixer_ops.sigmoid_topk(mixer_ops.router_logits(x, w), top)
    assert torch.equal(ids, want) and torch.equal(weights.view(torch.int32), want_w.view(torch.int32))


@pytest.mark.parametrize("E", [1, 8, 48])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 1023, 1024, 1025, 2047, 8198, 16383, 16384])
def test_expert_order(n, E):
    gen = torch.Generator(device="cuda").manual_seed(n)
    ids = torch.randint(0, E, (n, 1), generator=gen, device="cuda", dtype=torch.int32)
    if n > 40:
        ids[5], ids[17] = -3, E + 2                  # of no expert: behind the last
    order, where, offsets = mixer_ops.expert_order(ids, E)
    key = torch.where((ids[:, 0] < 0) | (ids[:, 0] >= E), E, ids[:, 0]).to(torch.int64)
    want = torch.sort(key, stable=True).indices
    assert torch.equal(order, want) and torch.equal(where[order], torch.arange(n, device="cuda"))
    assert torch.equal(offsets.long(), torch.searchsorted(key[want], torch.arange(E + 1, device="cuda")))


@pytest.mark.parametrize("E,launches", [(8, ["_router_sigmoid_topk"]), (12, ["router_logits", "sigmoid_topk"])])
def test_every_launch_is_timed_once(E, launches, monkeypatch):
    monkeypatch.setattr(mixer_ops, "EVENTS", [])
    mixer_ops.router_sigmoid_topk(torch.randn(5, 64, device="cuda"), torch.randn(E, 64, device="cuda"), 2)
    assert [name for name, _a, _b in mixer_ops.EVENTS] == launches
