"""Rotary rows in 16-byte pieces (q and k with norm, rotation and append; latent rows) and value rows, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F64, EPS = torch.float64, 1e-5


def _turn(x, pos, freqs, interleaved):
    half = len(freqs)
    ang = pos.to(F64)[:, None, None] * freqs
    c, s = ang.cos(), ang.sin()
    y = x.clone()
    a, b = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if interleaved else (slice(0, half), slice(half, 2 * half))
    u, v = x[..., a], x[..., b]
    y[..., a], y[..., b] = u * c - v * s, v * c + u * s
    return y


def _unit(x):
    return x * (x.square().mean(-1, keepdim=True) + EPS).rsqrt()


def _near(got, want, dtype, turned):
    # one rounding to the storage type of a value of at most `turned` (a turned pair mixes both members), beside fp32's own
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert ((got.to(F64) - want).abs() <= eps * want.abs() + 4e-6 * turned).all()


def _slots(n, bs):
    slots = torch.randperm((n // bs + 1) * bs, device="cuda")[:n]
    slots[n // 2] = -1
    return slots


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,H,G,dk,dv,rot,interleaved,norm", [
    (1, 3, 1, 64, 64, 16, 0, 1), (593, 2, 1, 128, 72, 128, 0, 1), (1187, 1, 1, 256, 8, 24, 1, 0), (2371, 3, 2, 64, 128, 64, 1, 1), (37, 5, 2, 128, 128, 0, 0, 1)])
def test_q_and_k(n, H, G, dk, dv, rot, interleaved, norm, dtype):
    from dgi_b200 import mixer_ops
    torch.manual_seed(n)
    bs = 16
    wide = torch.randn(n, (H + G) * dk + G * dv + 8, device="cuda").to(dtype)
    q, k, v = wide[:, :H * dk], wide[:, H * dk:(H + G) * dk], wide[:, (H + G) * dk:(H + G) * dk + G * dv]
    w = [(1 + 0.2 * torch.randn(dk, device="cuda")).to(dtype) if norm else None for _ in range(2)]
    freqs = torch.rand(rot // 2, dtype=F64, device="cuda")
    pos, slots = torch.randint(0, 70000, (n,), dtype=torch.int32, device="cuda"), _slots(n, bs)
    want = []
    for x, heads, wt in ((q, H, w[0]), (k, G, w[1])):
        y = x.to(F64).view(n, heads, dk)
        want.append(_turn(_unit(y) * wt.to(F64) if norm else y, pos, freqs, interleaved))
    kp = torch.full((n // bs + 1, G, bs, dk), float("nan"), dtype=dtype, device="cuda")
    vp = torch.full((n // bs + 1, G, bs, dv), float("nan"), dtype=dtype, device="cuda")
    mixer_ops.qknorm_rotary_append(q, k, v, *w, EPS, freqs if rot else None, kp, vp, slots, pos, H, interleaved=bool(interleaved))
    top = max(x.abs().max().item() for x in want)
    _near(q.view(n, H, dk), want[0], dtype, top)
    live = slots >= 0
    s = slots[live]
    _near(kp[s // bs, :, s % bs], want[1][live], dtype, top)
    assert torch.equal(vp[s // bs, :, s % bs], v.view(n, G, dv)[live])
    assert int((~kp.isnan().any(-1)).sum()) == int(live.sum()) * G                 # nothing beside the slots was written


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,H,rank,dr,rot,interleaved", [(1, 2, 8, 16, 16, 0), (593, 1, 264, 64, 32, 0), (1187, 3, 512, 24, 24, 1), (2371, 2, 256, 64, 64, 1), (21, 2, 40, 8, 0, 1)])
def test_latents(n, H, rank, dr, rot, interleaved, dtype):
    from dgi_b200 import mixer_ops
    torch.manual_seed(n)
    bs, gain = 16, 1.25
    wide = torch.randn(n, H * (16 + dr) + rank + dr, device="cuda").to(dtype)
    q, dkv = wide[:, :H * (16 + dr)].unflatten(1, (H, 16 + dr)), wide[:, H * (16 + dr):]
    w = (1 + 0.2 * torch.randn(rank, device="cuda")).to(dtype)
    freqs = torch.rand(rot // 2, dtype=F64, device="cuda")
    pos, slots = torch.randint(0, 70000, (n,), dtype=torch.int32, device="cuda"), _slots(n, bs)
    pool = torch.full((n // bs + 1, 1, bs, rank + dr), float("nan"), dtype=dtype, device="cuda")
    out = torch.full((n, H, rank + dr), float("nan"), dtype=dtype, device="cuda")
    mixer_ops.latent_rotary_append(q[:, :, 16:], out[:, :, rank:], dkv, w, EPS, freqs if rot else None, gain, pool, slots, pos, interleaved=bool(interleaved))

    def turned(x):
        y = _turn(x, pos, freqs, interleaved)
        y[..., :rot] *= gain
        return y

    want_q, want_k = turned(q[:, :, 16:].to(F64)), turned(dkv[:, None, rank:].to(F64))[:, 0]
    want_c = _unit(dkv[:, :rank].to(F64)) * w.to(F64)
    top = max(x.abs().max().item() for x in (want_q, want_k, want_c))
    _near(out[:, :, rank:], want_q, dtype, top)
    live = slots >= 0
    rows = pool.view(-1, rank + dr)[slots[live]]
    _near(rows[:, :rank], want_c[live], dtype, top)
    _near(rows[:, rank:], want_k[live], dtype, top)
    assert int((~pool.isnan().any(-1)).sum()) == int(live.sum()) and out[:, :, :rank].isnan().all()


@pytest.mark.parametrize("n,G,dk,dv", [(1, 1, 8, 64), (9, 3, 64, 256), (1001, 1, 200, 128), (70, 5, 136, 64)])
def test_values(n, G, dk, dv):
    from dgi_b200 import mixer_ops
    torch.manual_seed(n)
    bs, dtype = 16, torch.bfloat16
    wide = torch.randn(n, G * (dk + dv), device="cuda").to(dtype)
    k, v = wide[:, :G * dk], wide[:, G * dk:]
    prev, keep, slots = torch.randn(n, G * dv, device="cuda").to(dtype), torch.empty(n, G * dv, device="cuda", dtype=dtype), _slots(n, bs)
    kp = torch.full((n // bs + 1, G, bs, dk), float("nan"), dtype=dtype, device="cuda")
    vp = torch.full((n // bs + 1, G, bs, dv), float("nan"), dtype=dtype, device="cuda")
    mixer_ops.value_prep_append(k, v, kp, vp, slots, EPS, v_prev=prev, lam=0.3, v_keep=keep)
    want = 0.7 * _unit(v.to(F64).view(n, G, dv)) + 0.3 * prev.to(F64).view(n, G, dv)
    _near(keep.view(n, G, dv), want, dtype, want.abs().max().item())
    s = slots[slots >= 0]
    assert torch.equal(kp[s // bs, :, s % bs], k.view(n, G, dk)[slots >= 0]) and torch.equal(vp[s // bs, :, s % bs], keep.view(n, G, dv)[slots >= 0])
    assert int((~kp.isnan().any(-1)).sum()) == len(s) * G
