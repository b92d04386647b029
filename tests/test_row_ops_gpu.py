"""Row kernels at the edges of their register tiles (a piece of eight per lane, one, four or eight warps per row) and off the 16-byte
grid, and the one-CTA expert order around its chunk sizes."""
import pytest
import torch

from dgi_b200 import mixer_ops

pytestmark = pytest.mark.gpu

F64 = torch.float64
EPS = 1e-5
WIDTHS = [8, 64, 504, 512, 520, 1024, 1032, 2048, 4088, 4104, 8192, 8200, 16384, 16392, 1, 30, 1001]
TOL = {torch.float32: 2e-6, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -10}     # one rounding of the result; fp32: its own sums


def _unit(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _close(got, want, dtype):
    return ((got.to(F64) - want).abs() <= TOL[dtype] * (want.abs() + want.square().mean().sqrt())).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("width", WIDTHS)
def test_norms_and_polynorm(width, dtype):
    gen = torch.Generator(device="cuda").manual_seed(width)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    rows = 5
    x, w, w2 = rnd(rows, width) * 3, (rnd(width) * 0.2).to(dtype), (rnd(width) * 0.2).to(dtype)
    assert _close(mixer_ops.offset_rmsnorm(x, w, EPS), _unit(x.to(F64)) * (1 + w.to(F64)), dtype)
    y = rnd(rows, width + 8).to(dtype)[:, :width]                       # rows of a wider projection
    new = x.to(F64) + 0.7 * _unit(y.to(F64)) * (1 + w.to(F64))
    out = mixer_ops.postnorm_residual(x, y, w, 0.7, EPS, w_next=w2)
    assert _close(x, new, torch.float32)
    assert _close(out, _unit(new) * (1 + w2.to(F64)), dtype)
    coef = torch.tensor([0.6, 0.3, -0.2, 0.05], device="cuda").to(dtype)
    z, c = y.to(F64), coef.to(F64)
    assert _close(mixer_ops.polynorm(y, coef, EPS), c[0] * _unit(z) + c[1] * _unit(z * z) + c[2] * _unit(z ** 3) + c[3], dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("G,dk,dv,odd", [(4, 128, 128, 0), (1, 16, 260, 0), (3, 30, 7, 0), (2, 64, 64, 1), (5, 132, 4, 0)])
def test_value_prep(G, dk, dv, odd, dtype):
    gen = torch.Generator(device="cuda").manual_seed(G * dk)
    n, bs = 9, 4
    wide = torch.randn(n, G * (dk + dv) + 8 + odd, generator=gen, device="cuda").to(dtype)
    k, v = wide[:, odd:odd + G * dk], wide[:, odd + G * dk:odd + G * (dk + dv)]
    kp, vp = torch.zeros(4, G, bs, dk, device="cuda", dtype=dtype), torch.zeros(4, G, bs, dv, device="cuda", dtype=dtype)
    slots = torch.tensor([15, 0, -1, 7, 3, 16, 9, 10, 2], device="cuda")     # one unused, one beyond the pool
    prev, keep = torch.randn(n, G * dv, generator=gen, device="cuda").to(dtype), torch.empty(n, G * dv, device="cuda", dtype=dtype)
    mixer_ops.value_prep_append(k, v, kp, vp, slots, EPS, v_prev=prev, lam=0.3, v_keep=keep)
    want = 0.7 * _unit(v.to(F64).reshape(n, G, dv)) + 0.3 * prev.to(F64).view(n, G, dv)
    assert _close(keep.view(n, G, dv), want, dtype)
    for i, s in enumerate(slots.tolist()):
        if 0 <= s < 16:
            assert torch.equal(kp[s // bs, :, s % bs], k[i].view(G, dk)) and torch.equal(vp[s // bs, :, s % bs], keep[i].view(G, dv))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("dv", [128, 4, 512, 132, 516, 33])
def test_head_norm(dv, dtype):
    x = torch.randn(11, 3, dv, device="cuda")
    w = (1 + 0.1 * torch.randn(dv, device="cuda")).to(dtype)
    assert _close(mixer_ops.head_rmsnorm(x, w, EPS), _unit(x.to(F64)) * w.to(F64), dtype)


@pytest.mark.parametrize("n,top,E", [(1, 1, 1), (5, 3, 7), (512, 2, 8), (513, 2, 8), (4099, 2, 48), (8192, 2, 5), (8193, 2, 5), (1000, 4, 49), (70000, 2, 3)])
def test_expert_order(n, top, E):
    ids = torch.randint(0, E, (n, top), dtype=torch.int32, device="cuda")
    if E > 2:
        ids[ids == 1] = 0                                             # an expert without rows
    order, where, offsets = mixer_ops.expert_order(ids, E)
    want = torch.argsort(ids.reshape(-1), stable=True)
    assert torch.equal(order, want) and torch.equal(where[order], torch.arange(n * top, device="cuda"))
    assert offsets.tolist() == [0] + torch.bincount(ids.reshape(-1), minlength=E).cumsum(0).tolist()


@pytest.mark.parametrize("n,top,E", [(7, 2, 5), (513, 2, 48), (700, 2, 49), (70000, 2, 3)])
def test_expert_order_is_a_permutation_whatever_the_ids(n, top, E):
    """Pairs of no expert come behind the last one: rows are addressed by ``order`` and ``where``."""
    gen = torch.Generator().manual_seed(n)
    ids = torch.randint(0, E, (n, top), dtype=torch.int32, generator=gen)
    ids[::3, 0] = 0x7fffffff
    ids[1::5, 1] = -1
    ids[2::7, 0] = E
    flat = torch.where((ids < 0) | (ids >= E), E, ids).reshape(-1)
    want = torch.argsort(flat, stable=True)
    order, where, offsets = (t.cpu() for t in mixer_ops.expert_order(ids.cuda(), E))
    assert torch.equal(order, want) and torch.equal(where, torch.argsort(want))
    assert offsets.tolist() == [0] + torch.bincount(flat, minlength=E + 1)[:E].cumsum(0).tolist()


def test_sigmoid_topk_names_experts_for_tokens_of_nans():
    nan, inf = float("nan"), float("inf")
    rows = [[nan] * 40, [nan] * 39 + [1.0], [-inf] * 40, [0.0] * 20 + [nan] * 20, [nan, -inf] * 20]
    ids, w = (t.cpu() for t in mixer_ops.sigmoid_topk(torch.tensor(rows, device="cuda"), 3))
    assert ids.tolist() == [[0, 1, 2], [39, 0, 1], [0, 1, 2], [0, 1, 2], [1, 3, 5]]
    assert w[0].isnan().all() and w[1, 1:].isnan().all()
    assert abs(w[1, 0].item() - 1 / (1 + 2.718281828459045 ** -1)) < 2.0 ** -22      # e^-1, a sum and a quotient, each rounded once or twice
    assert (w[2] == 0).all() and (w[3] == 0.5).all() and (w[4] == 0).all()


@pytest.mark.parametrize("groups,keep", [(1, 1), (4, 2)])
@pytest.mark.parametrize("scores", ["softmax", "sigmoid"])
def test_group_topk_names_experts_for_tokens_of_nans(scores, groups, keep):
    E, top, nan = 40, 3, float("nan")
    gen = torch.Generator(device="cuda").manual_seed(E)
    z = torch.randn(6, E, generator=gen, device="cuda")
    plain = z.clone()
    z[1], z[3] = nan, nan
    z[4, 5:] = nan
    call = {"softmax": lambda x: mixer_ops.softmax_group_topk(x, None, top, groups, keep, sum_floor=1e-9),
            "sigmoid": lambda x: mixer_ops.sigmoid_group_topk(x, None, E, top, groups, keep)}[scores]
    (ids, w), (ids0, w0) = call(z), call(plain)
    assert ((ids >= 0) & (ids < E)).all() and all(len(set(r)) == top for r in ids.tolist())
    assert w[[1, 3]].isnan().all()
    for r in (0, 2, 5):
        assert torch.equal(ids[r], ids0[r]) and torch.equal(w[r], w0[r])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("n", [9, 1500])
def test_a_token_of_nans_stays_its_own(n, dtype):
    """Routed experts, the grouped kernel's sizes and the library's: the other tokens' rows are what they are without it."""
    from dgi_b200.petipel_layer import SigmoidTopKMoE

    gen = torch.Generator(device="cuda").manual_seed(n)
    E, W, ff = 5, 64, 32
    lin = lambda o, i: torch.randn(o, i, generator=gen, device="cuda") / i ** 0.5  # noqa: E731
    t = {f"e{e}.{k}": lin(*s) for e in range(E) for k, s in (("gate", (ff, W)), ("up", (ff, W)), ("down", (W, ff)))}
    moe = SigmoidTopKMoE({"router": {"experts": E, "top": 2}, "expert": {"limit": 7.0}}, dict(t, router=lin(E, W)), "cuda", dtype)
    h = torch.randn(n, W, generator=gen, device="cuda").to(dtype)
    bad = h.clone()
    bad[4] = float("nan")
    out, want = moe(bad), moe(h)
    rest = torch.arange(n, device="cuda") != 4
    # another token's pairs move to other rows of the same products: their sums keep their order, or differ by its rounding
    assert ((out - want)[rest].norm() / want[rest].norm()) <= {torch.float32: 1e-6}.get(dtype, 4 * TOL[dtype])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("width", [8, 1024, 1032, 100])
def test_expert_rows(width, dtype):
    n, top, E = 37, 2, 5
    h, wts = torch.randn(n, width, device="cuda").to(dtype), torch.rand(n, top, device="cuda")
    order, where, _ = mixer_ops.expert_order(torch.randint(0, E, (n, top), dtype=torch.int32, device="cuda"), E)
    xs = mixer_ops.scaled_gather(h, wts.reshape(-1), order, top)
    assert _close(xs, wts.reshape(-1)[order].to(F64)[:, None] * h.to(F64)[order // top], dtype)
    g, u = (xs.to(F64)[:, i * (width // 2):(i + 1) * (width // 2)] for i in range(2))
    g, u = g.clamp(max=0.8), u.clamp(-0.8, 0.8)
    assert _close(mixer_ops.clamped_glu(xs, 0.8, 1.7), g * torch.sigmoid(1.7 * g) * (u + 1), dtype)
    assert _close(mixer_ops.expert_combine(xs, where, n, top), xs.to(F64)[where].view(n, top, width).sum(1), torch.float32)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("B,T,D,scaling", [(1, 1, 2, 1.0), (4, 1, 64, 1.0), (3, 7, 128, 1.2), (1, 300, 96, 1.0)])
def test_rope_tables(B, T, D, scaling, dtype):
    from dgi_b200 import paged_layer

    pos = torch.randint(0, 100000, (B, T), device="cuda")
    inv = 10000.0 ** (-torch.arange(0, D, 2, device="cuda", dtype=torch.float32) / D)
    ang = pos.to(torch.float32)[:, :, None] * inv
    ang = torch.cat((ang, ang), dim=-1)
    cos, sin = paged_layer.rope_tables(pos, inv, dtype, scaling)
    want = [(f * scaling).to(dtype) if scaling != 1.0 else f.to(dtype) for f in (ang.cos(), ang.sin())]
    assert torch.equal(cos, want[0]) and torch.equal(sin, want[1])     # the same fp32 operations, rounded once


@pytest.mark.parametrize("layers,blocks,slots", [(1, 3, [1]), (33, 700, list(range(0, 700, 1))), (2, 50, [49, 0, 7])])
def test_zero_blocks(layers, blocks, slots):
    pools = [torch.ones(blocks, 2, 4, 8 * (1 + i % 3), device="cuda", dtype=torch.bfloat16) for i in range(layers)]
    mixer_ops.zero_blocks(pools, slots)
    for p in pools:
        assert (p[slots] == 0).all() and p.float().sum() == (blocks - len(slots)) * p[0].numel()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("dv,odd", [(128, 0), (8, 0), (72, 0), (256, 0), (264, 0), (512, 0), (516, 0), (33, 0), (128, 1)])
@pytest.mark.parametrize("weight,gate,act", [(True, True, "sigmoid"), (False, True, "silu"), (False, False, "sigmoid")])
def test_gated_head_norm(dv, odd, weight, gate, act, dtype):
    n, H = 7, 5                                                        # 35 rows: the last warp's are cut short
    x = torch.randn(n, H, dv, device="cuda")
    w = (1 + 0.1 * torch.randn(dv, device="cuda")).to(dtype) if weight else None
    g = torch.randn(n, H * dv + 8 + odd, device="cuda").to(dtype)[:, odd:odd + H * dv] if gate else None
    g64 = g.to(F64).reshape(n, H, dv) if gate else None
    want = _unit(x.to(F64)) * (w.to(F64) if weight else 1)
    gated = want if not gate else want * torch.sigmoid(g64) * (g64 if act == "silu" else 1)
    got = mixer_ops.head_norm_act_gate(x, w, g, EPS, dtype, gate_act=act, out_scale=-0.7)
    assert _close(got.view(n, H, dv), -0.7 * gated, dtype)
    if weight:
        got = mixer_ops.head_rmsnorm_gated(x, w, g, EPS)
        assert _close(got.view(n, H, dv), gated, dtype)


@pytest.mark.parametrize("dtype,C", [(torch.bfloat16, 8), (torch.bfloat16, 7), (torch.float32, 6)])
@pytest.mark.parametrize("taps", [1, 4, 6, 16])
@pytest.mark.parametrize("cuts", [(1, 1, 2, 1, 9), (8, 7, 3), (64, 1, 65), (130,)])
def test_causal_conv_portions(cuts, taps, dtype, C):
    x, w = torch.randn(sum(cuts), C, device="cuda").to(dtype), torch.randn(C, taps, device="cuda").to(dtype)
    tail, got, at = torch.full((2, taps - 1, C), 9.0, device="cuda"), [], 0
    for cut in cuts:
        seqs = torch.tensor([[0, cut, 1, int(at == 0)]], dtype=torch.int32, device="cuda")
        got.append(mixer_ops.causal_conv_silu(x[at:at + cut], w, tail, seqs, cut))
        at += cut
    pad = torch.cat((torch.zeros(taps - 1, C, device="cuda", dtype=F64), x.to(F64)))
    y = sum(pad[i:i + sum(cuts)] * w[:, i].to(F64) for i in range(taps))
    tol = {torch.bfloat16: 2.0 ** -8, torch.float32: 4e-6}[dtype]       # taps products of up to ~ 10, then one rounding
    assert ((torch.cat(got).to(F64) - y * torch.sigmoid(y)).abs() <= tol * (y.abs() + 1)).all()


def test_launches_of_different_sizes_from_two_threads():
    """One kernel, dynamic shared memory by the call: another thread's smaller launch must not lower the limit in between."""
    import threading

    ids = {E: torch.randint(0, E, (500, 2), dtype=torch.int32, device="cuda") for E in (13, 24, 40, 48)}
    torch.cuda.synchronize()      # the threads' streams start from here
    failed = []

    def work(sizes):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for i in range(1500):
                    E = sizes[i % 2]
                    last = mixer_ops.expert_order(ids[E], E)
                assert torch.equal(last[0], torch.argsort(ids[E].reshape(-1), stable=True))
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in ((13, 48), (40, 24), (48, 40), (13, 24))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("width", [64, 1032, 30])
def test_rows_of_nans_and_infinities_stay_their_own(width, dtype):
    gen = torch.Generator(device="cuda").manual_seed(width)
    x = torch.randn(6, width, generator=gen, device="cuda")
    w = (torch.randn(width, generator=gen, device="cuda") * 0.2).to(dtype)
    coef = torch.tensor([0.6, 0.3, -0.2, 0.05], device="cuda").to(dtype)
    bad = x.clone()
    bad[1], bad[3, 2] = float("nan"), float("inf")
    rest = [0, 2, 4, 5]
    for op in (lambda v: mixer_ops.offset_rmsnorm(v, w, EPS), lambda v: mixer_ops.polynorm(v.to(dtype), coef, EPS),
               lambda v: mixer_ops.head_rmsnorm(v.view(6, 1, width), w, EPS).view(6, -1),
               lambda v: mixer_ops.postnorm_residual(v.clone(), v.to(dtype), w, 0.7, EPS, w_next=w)):
        got, want = op(bad), op(x)
        assert torch.equal(got[rest], want[rest]) and got[1].isnan().all() and got[3, 2].isnan()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("n", [1, 9, 1023, 1500])
def test_routed_experts_of_every_path(n, dtype):
    """The grouped kernel up to 2048 pairs, beyond it the library's grouped GEMM (bf16) or one GEMM per expert (fp16, fp32)."""
    from dgi_b200.petipel_layer import SigmoidTopKMoE

    gen = torch.Generator(device="cuda").manual_seed(n)
    E, W, ff, limit = 5, 64, 32, 1.5
    lin = lambda o, i: (torch.randn(o, i, generator=gen, device="cuda") / i ** 0.5).to(dtype)  # noqa: E731
    t = {f"e{e}.{k}": lin(*s) for e in range(E) for k, s in (("gate", (ff, W)), ("up", (ff, W)), ("down", (W, ff)))}
    t["router"] = lin(E, W)
    moe = SigmoidTopKMoE({"router": {"experts": E, "top": 2}, "expert": {"limit": limit}}, t, "cuda", dtype)
    h = torch.randn(n, W, generator=gen, device="cuda").to(dtype)
    z = h.to(F64) @ t["router"].to(F64).T
    top, ids = z.topk(2, dim=1)
    want = torch.zeros(n, W, dtype=F64, device="cuda")
    for k in range(2):
        for e in range(E):
            rows = ids[:, k] == e
            xs = (torch.sigmoid(top[rows, k])[:, None] * h[rows].to(F64)).to(dtype).to(F64)
            g = (xs @ t[f"e{e}.gate"].to(F64).T).clamp(max=limit)
            u = (xs @ t[f"e{e}.up"].to(F64).T).clamp(-limit, limit)
            want[rows] += (g * torch.sigmoid(1.702 * g) * (u + 1)) @ t[f"e{e}.down"].to(F64).T
    # inputs, products, activations and outputs of an expert each rounded once
    assert (moe(h) - want).norm() / want.norm() <= {torch.float32: 2e-6}.get(dtype, 4 * TOL[dtype])
