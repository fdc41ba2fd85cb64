"""Row kernels that move 16 bytes at a time, at the edges of what they take, against 64-bit.

Tolerances: a bfloat16 result is off by its rounding, 2^-8 of it, beside a 32-bit sum of n terms, n * 2^-24 of
itself at most, and the 32-bit functions (exp, sin, rsqrt and products), 2^-20 of it taken together.
"""
import pytest
import torch

from atom_b200 import native

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rand(*shape, dtype=torch.bfloat16, seed=0):
    g = torch.Generator(device="cpu").manual_seed(seed + sum(shape))
    return torch.randn(*shape, generator=g).to(DEV, dtype)


def shifted(x, by):
    """The same numbers, ``by`` numbers behind a 16-byte boundary."""
    buf = torch.empty(x.numel() + by, dtype=x.dtype, device=x.device)
    buf[by:].copy_(x.reshape(-1))
    return buf[by:].view(x.shape)


def norm64(x, w, eps):
    x = x.double()
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()


def close(got, want, n):
    rel = (2.0 ** -8 if got.dtype == torch.bfloat16 else 0.0) + n * 2.0 ** -24 + 2.0 ** -20
    assert bool(((got.double() - want).abs() <= rel * want.abs() + 1e-6).all())


@pytest.mark.parametrize("n,by,wd", [(8, 0, torch.float32), (264, 0, torch.bfloat16), (4096, 0, torch.bfloat16),
                                     (4104, 0, torch.float32), (8192, 0, torch.bfloat16), (8200, 0, torch.bfloat16),
                                     (1030, 0, torch.bfloat16), (1024, 4, torch.bfloat16)])
def test_norms_of_whole_rows(n, by, wd):
    T = 5
    seq = torch.tensor([0, 0, -1, 1, 1], dtype=torch.int32, device=DEV)
    a, b, c = (shifted(rand(T, n, seed=i), by) for i in range(3))
    wa, wb = rand(n, dtype=wd, seed=3), rand(n, dtype=wd, seed=4)
    for parts in ((wa, b, wb, c), (wa, b, wb, None), (wa, None, None, c), (None, None, None, c)):
        x, y, z, u = parts
        res = rand(T, n, dtype=torch.float32, seed=5)
        want = norm64(a, x, 1e-6) if x is not None else a.double()
        if y is not None:
            want = 0.5 * (want + norm64(y, z, 1e-6))
        want = res.double() + want + (u.double() if u is not None else 0.0)
        sizes = 4.0 + res.abs().double()        # (the terms may cancel: errors are of the terms' size)
        native.pair_rmsnorm_add(res, a, x, y, z, u, 1e-6)
        assert bool(((res.double() - want).abs() <= (n * 2.0 ** -24 + 2.0 ** -20) * (sizes + want.abs()) * 4).all())
    o, proj = rand(T, n, dtype=torch.float32, seed=6), shifted(rand(T, 3 * n, seed=7), by)
    out = torch.full((T, n), 7.0, dtype=torch.bfloat16, device=DEV)
    gate = proj[:, n:2 * n]
    native.lightning_gate_norm(out, o, gate, wa, 1e-6, seq)
    live = seq >= 0
    close(out[live], (norm64(o, wa, 1e-6) * torch.sigmoid(gate.double()))[live], n)
    assert bool((out[~live] == 7.0).all())


@pytest.mark.parametrize("rq,r,rd,dims,by", [(8, 8, 8, 8, 0), (0, 512, 64, 64, 0), (264, 72, 24, 16, 0), (3584, 512, 64, 64, 0),
                                             (3592, 520, 64, 32, 0), (8192, 512, 64, 64, 0), (96, 40, 12, 12, 0),
                                             (96, 40, 16, 16, 4)])
def test_latents_and_rotated_keys(rq, r, rd, dims, by):
    T, ps = 6, 4
    seq = torch.tensor([0, 0, 0, 1, -1, 2], dtype=torch.int32, device=DEV)
    pos = torch.tensor([3, 4, 5, 900, 0, 0], dtype=torch.int32, device=DEV)
    table = torch.zeros(3, 226, dtype=torch.int32, device=DEV)
    table[0, 0], table[0, 1], table[1, 225], table[2, 0] = 2, 0, 1, 77       # (77: no such page)
    proj = shifted(rand(T, rq + r + rd + 8), by)
    wq, wkv = (rand(rq, seed=1) if rq else None), rand(r, seed=2)
    freq = torch.rand(max(dims // 2, 1), device=DEV)
    pages = torch.full((3, ps, r + rd), 7.0, dtype=torch.bfloat16, device=DEV)
    cq = torch.full((T, rq), 7.0, dtype=torch.bfloat16, device=DEV) if rq else None
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    native.latent_prepare(cq, proj, 0, wq, 1e-6, pos, seq, rq, r, rd, dims, wkv, freq, 0.5, table, ps, pages, status)
    live = seq >= 0
    if rq:
        close(cq[live], norm64(proj[:, :rq], wq, 1e-6)[live], rq)
        assert bool((cq[~live] == 7.0).all())
    assert int(status) == 1
    keys = proj[:, rq + r:rq + r + rd].double()
    angle = (pos.float()[:, None] * freq[: dims // 2]).double()
    cos, sin = 0.5 * angle.cos(), 0.5 * angle.sin()
    half = dims // 2
    lo, hi = keys[:, :half], keys[:, half:dims]
    rot = torch.cat([lo * cos - hi * sin, hi * cos + lo * sin, keys[:, dims:]], 1)
    latent = norm64(proj[:, rq:rq + r], wkv, 1e-6)
    used = torch.zeros(3, ps, dtype=torch.bool)
    for t, (page, slot) in enumerate([(2, 3), (0, 0), (0, 1), (1, 0)]):
        used[page, slot] = True
        close(pages[page, slot, :r], latent[t], r)
        want = rot[t]
        size = torch.cat([(lo * cos).abs() + (hi * sin).abs(), (hi * cos).abs() + (lo * sin).abs(), keys[:, dims:].abs()], 1)[t]
        assert bool(((pages[page, slot, r:].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20 * size).all())
    assert bool((pages[~used] == 7.0).all())


@pytest.mark.parametrize("W,by,mud", [(8, 0, torch.bfloat16), (520, 0, torch.float32), (4104, 0, torch.bfloat16),
                                      (1024, 4, torch.bfloat16), (36, 0, torch.float32)])
def test_token_shift(W, by, mud):
    T, n = 7, 5
    seq = torch.tensor([0, 0, 0, 1, 2, 2, -1], dtype=torch.int32, device=DEV)
    cu = torch.tensor([0, 3, 4, 6], dtype=torch.int32, device=DEV)
    slots = torch.tensor([2, 0, 3], dtype=torch.int32, device=DEV)
    h, mu, state = rand(T, W), shifted(rand(n, W, dtype=mud, seed=1), by), rand(4, W, seed=2)
    old = state.clone()
    out = torch.full((n, T, W), 7.0, dtype=torch.bfloat16, device=DEV)
    native.token_shift_mix(out, h, mu, state, seq, cu, slots)
    prev = torch.cat([old[2:3], h[0:2], old[0:1], old[3:4], h[4:5]]).double()
    cur = h[:6].double()
    want = cur + (prev - cur) * mu.double()[:, None]
    size = cur.abs() + (prev - cur).abs() * mu.double().abs()[:, None]
    assert bool(((out[:, :6].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -22 * size).all())
    assert bool((out[:, 6] == 7.0).all())
    assert torch.equal(state[[2, 0, 3]], h[[2, 3, 5]]) and torch.equal(state[1], old[1])


@pytest.mark.parametrize("n,rows,wd", [(8, 5, torch.float32), (264, 5, torch.bfloat16), (1024, 5, torch.float32), (2048, 5, torch.bfloat16),
                                       (4096, 5, torch.float32), (256, 8195, torch.bfloat16), (512, 4096, torch.float32),
                                       (768, 2733, torch.bfloat16), (1536, 1365, torch.float32), (1536, 1368, torch.bfloat16),
                                       (2048, 1023, torch.bfloat16), (2048, 1024, torch.float32), (2560, 1022, torch.bfloat16),
                                       (3584, 601, torch.float32), (4096, 512, torch.float32), (4096, 515, torch.bfloat16)])
def test_mean_of_two_norms(n, rows, wd):
    """Few numbers and many (from 2^21 on whole warps take rows of a multiple of 256)."""
    a, b, wa, wb = rand(rows, n), rand(rows, n, seed=1), rand(n, dtype=wd, seed=2), rand(n, dtype=wd, seed=3)
    out = torch.empty(rows, n, dtype=torch.bfloat16, device=DEV)
    assert native.pair_rmsnorm_takes(out, a, wa, b, wb)
    native.pair_rmsnorm(out, a, wa, b, wb, 1e-5)
    close(out, 0.5 * (norm64(a, wa, 1e-5) + norm64(b, wb, 1e-5)), n)


def test_what_the_mean_of_two_norms_does_not_take():
    a, w = rand(5, 1024), rand(1024)
    out = torch.empty_like(a)
    assert not native.pair_rmsnorm_takes(shifted(out, 4), a, w, a, w) and not native.pair_rmsnorm_takes(out, a, w, a, w.float())
    assert not native.pair_rmsnorm_takes(out.float(), a.float(), w, a.float(), w) and not native.pair_rmsnorm_takes(out, rand(5, 4104), w, a, w)
    with pytest.raises(native.NativeError):
        native.pair_rmsnorm(shifted(out, 4), a, w, a, w, 1e-5)


@pytest.mark.parametrize("M,N,K", [(9, 151936, 64), (16, 128256, 192), (13, 75777, 128)])
def test_products_of_few_rows_with_a_matrix_as_tall_as_a_head(M, N, K):
    """More sub-slabs of W's rows a CTA than eight, the last of them cut short: 32-bit sums of K products of bfloat16 numbers lie
    within K 2^-24 of the sums of their magnitudes."""
    g = torch.Generator(device="cuda:0").manual_seed(N)
    x = torch.randn(M, K, device="cuda:0", generator=g).to(torch.bfloat16)
    w = torch.randn(N, K, device="cuda:0", generator=g).to(torch.bfloat16)
    out = torch.full((M, N), float("nan"), device="cuda:0")
    assert native.gemm_rows_supports(M, N, K, K)
    native.gemm_rows(x, w, out)
    off = (out.double() - x.double() @ w.double().T).abs()
    assert bool((off <= K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)).all())
