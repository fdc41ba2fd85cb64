"""Attention of prompt portions on tcgen05 (csrc/window_prefill_tc.cu) against 64-bit: windows, chunks and all keys, one map and two,
sinks and gates, paged keys and keys in arrays with a shared part, requests at the edges of tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
F64 = torch.float64
Q_LENS = [([64], [0]), ([1, 130, 3, 257], [700, 0, 64, 31]), ([500, 1, 40], [1000, 127, 128])]


def _rel(got, want):
    return float((got.double().cpu() - want).norm() / want.norm())


def _seen(start, n, window, chunked):
    pos, key = torch.arange(start, start + n)[:, None], torch.arange(start + n)[None]
    ok = key <= pos
    if window:
        ok &= (key // window == pos // window) if chunked else (key > pos - window)
    return ok


def _softmax(q, k, ok, scale, sink=None):
    s = (q @ k.T * scale).masked_fill(~ok, float("-inf"))
    if sink is not None:
        s = torch.cat([s, sink.expand(len(s), 1)], 1)
    return s.softmax(1)[:, : k.shape[0]]


def _arrays(q_lens, past):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    return i32([0] + torch.tensor(q_lens).cumsum(0).tolist()), i32([a + n for a, n in zip(past, q_lens)])


@pytest.mark.parametrize("q_lens,past", Q_LENS, ids=str)
@pytest.mark.parametrize("maps,window,chunked,group,page,extras", [
    (1, 0, False, 4, 16, False), (1, 200, False, 1, 8, True), (1, 128, True, 8, 64, True), (1, 1, False, 2, 128, True),
    (2, 0, False, 4, 16, False), (2, 300, True, 1, 16, True), (2, 64, False, 16, 32, False)])
def test_paged(q_lens, past, maps, window, chunked, group, page, extras):
    """Outputs are rounded to bfloat16 (2^-9); scores are sums of exact products, weights keep 16 bits."""
    from atom_b200 import native

    nkv, dk = 2, 128 // maps
    nh, T, scale = nkv * group, sum(q_lens), 1.5 * dk ** -0.5
    g = torch.Generator().manual_seed(group + window)
    bf = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)  # noqa: E731
    q, gate = bf(T, nh, maps, dk), bf(T, nh)
    sink = torch.randn(nh, generator=g) if extras and maps == 1 else None
    n_pages = [-(-(a + n) // page) for a, n in zip(past, q_lens)]
    perm = torch.randperm(sum(n_pages) + 3, generator=g).tolist()
    table = torch.full((len(q_lens), max(n_pages)), -1, dtype=torch.int32)
    kp, vp = bf(len(perm), nkv * maps, page, dk), bf(len(perm), nkv, page, 128)
    lam, eps, want, at = 0.4, 1e-5, torch.empty(T, nh, 128, dtype=F64), 0
    for i, (a, n) in enumerate(zip(past, q_lens)):
        table[i, : n_pages[i]] = torch.tensor([perm.pop() for _ in range(n_pages[i])], dtype=torch.int32)
        rows = table[i, : n_pages[i]].long()
        k = kp[rows].double().transpose(1, 2).reshape(-1, nkv, maps, dk)[: a + n]
        v = vp[rows].double().transpose(1, 2).reshape(-1, nkv, 128)[: a + n]
        ok = _seen(a, n, window, chunked)
        for h in range(nh):
            o = [_softmax(q[at:at + n, h, m].double(), k[:, h // group, m], ok, scale, sink[h].double() if sink is not None else None)
                 @ v[:, h // group] for m in range(maps)]
            if maps == 2:
                d = o[0] - lam * o[1]
                o = [d / (d.square().mean(1, keepdim=True) + eps).sqrt()]
            want[at:at + n, h] = o[0] * 0.7 * (torch.sigmoid(gate[at:at + n, h].double())[:, None] if extras else 1.0)
        # pages whose keys no row of the step sees have been given back
        first = int(ok.any(0).float().argmax())
        table[i, : first // page] = -1
        at += n
    cu, ctx = _arrays(q_lens, past)
    out = torch.full((T, nh * 128 + 8), float("nan"), dtype=torch.bfloat16, device=DEV)[:, : nh * 128]
    d = lambda t: t.to(DEV)  # noqa: E731
    assert native.lib().atom_window_prefill_supports(nh, nkv, dk, 128, maps, page)
    native.window_prefill(out, d(q.reshape(T, -1)), d(kp), d(vp), d(table), cu, ctx, len(q_lens), nh, nkv, dk, scale, window,
                          d(sink) if sink is not None else None, d(gate) if extras else None, 0.7, chunked, (lam, eps) if maps == 2 else None)
    native.check_error_flags()
    assert _rel(out.view(T, nh, 128), want) <= 3e-3


@pytest.mark.parametrize("q_lens,past", Q_LENS, ids=str)
@pytest.mark.parametrize("shared,window,heads", [(64, 0, 3), (64, 150, 16), (0, 1000, 5), (0, 0, 2)])
def test_keys_in_arrays_behind_a_latent(q_lens, past, shared, window, heads):
    """The rows that the step sees are copied out of the pages in the requests' order, queries are rotated in place."""
    from atom_b200 import native

    T, vec, R, page, scale = sum(q_lens), 128 + shared, 128, 16, 0.11
    g = torch.Generator().manual_seed(heads + window)
    bf = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)  # noqa: E731
    q, sink = bf(T, heads, vec + 8)[:, :, :vec].contiguous(), torch.randn(heads, generator=g)
    n_pages = [-(-(a + n) // page) for a, n in zip(past, q_lens)]
    perm = torch.randperm(sum(n_pages), generator=g).tolist()
    table, pages = torch.full((len(q_lens), max(n_pages)), -1, dtype=torch.int32), bf(len(perm), page, R + shared)
    freq = torch.rand(max(shared // 2, 1), generator=g)
    first = [max(0, a - window + 1) if window else 0 for a in past]
    keys = sum(a + n - f for a, n, f in zip(past, q_lens, first))
    rows, pos = [], torch.cat([torch.arange(a, a + n) for a, n in zip(past, q_lens)])
    for i, n in enumerate(n_pages):
        table[i, :n] = torch.tensor([perm.pop() for _ in range(n)], dtype=torch.int32)
        rows.append(pages[table[i, :n].long()].reshape(-1, R + shared)[first[i]: past[i] + q_lens[i]])
    d = lambda t: t.to(DEV)  # noqa: E731
    cu, ctx = _arrays(q_lens, past)
    dense, qd = torch.empty(keys, R + shared, dtype=torch.bfloat16, device=DEV), d(q)
    sot = torch.cat([torch.full((n,), i) for i, n in enumerate(q_lens)]).to(torch.int32).to(DEV)
    native.latent_expand(dense, d(pages), d(table), cu, ctx, len(q_lens), window, qd, 128, shared, d(freq), 1.25, d(pos.to(torch.int32)), sot)
    assert torch.equal(dense.cpu(), torch.cat(rows))
    if shared:
        h = shared // 2
        ang = pos[:, None].float() * freq
        c, s = (ang.cos() * 1.25)[:, None], (ang.sin() * 1.25)[:, None]
        a, b = q[..., 128:128 + h].float(), q[..., 128 + h:].float()
        want = torch.cat([q[..., :128].float(), a * c - b * s, b * c + a * s], -1)
        torch.testing.assert_close(qd.float().cpu(), want, rtol=8e-3, atol=8e-3)
    qr = qd.double().cpu()
    k, v = bf(keys, heads * 128), bf(keys, heads * 128)
    out = torch.full((T, heads, 128), float("nan"), dtype=torch.bfloat16, device=DEV)
    gate = bf(T, heads * 128) if window else None
    native.dense_prefill(out, qd, d(k), d(v), dense[:, R:] if shared else None, cu, ctx, len(q_lens), scale, window, d(sink),
                         d(gate) if window else None)
    native.check_error_flags()
    want, at, row = torch.empty(T, heads, 128, dtype=F64), 0, 0
    for a, n, f in zip(past, q_lens, first):
        ok, m = _seen(a, n, window, False)[:, f:], a + n - f
        for h in range(heads):
            kk = k[row:row + m, h * 128:(h + 1) * 128].double()
            if shared:
                kk = torch.cat([kk, dense[row:row + m, R:].double().cpu()], 1)
            want[at:at + n, h] = _softmax(qr[at:at + n, h], kk, ok, scale, sink[h].double()) @ v[row:row + m, h * 128:(h + 1) * 128].double()
        at, row = at + n, row + m
    if window:
        want *= torch.sigmoid(gate.double()).view(T, heads, 128)
    assert _rel(out, want) <= 3e-3


def _same_where_unseen(run, spoil, q_lens, past, window, chunked, column):
    """run() before and after spoil(): rows that see none of the spoilt numbers keep their results (up to one more rounding to
    bfloat16 on either side: 2^-7 of a number), a row that sees one of a value's shows it in that column."""
    clean = run().float().cpu()
    seen = spoil()                                    # per request: the spoilt key (-1: none)
    got = run().float().cpu()
    at = 0
    for a, n, key in zip(past, q_lens, seen):
        for t in range(n):
            pos = a + t
            low = 0 if not window else (pos // window * window if chunked else max(0, pos - window + 1))
            if low <= key <= pos:
                assert not bool(torch.isfinite(got[at + t, :, column]).any())
            else:
                torch.testing.assert_close(got[at + t], clean[at + t], rtol=2 ** -7, atol=2e-3)
        at += n


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("maps,window,chunked,group,page", [(1, 0, False, 4, 16), (1, 100, False, 1, 64), (2, 0, False, 2, 16),
                                                              (2, 64, True, 1, 32)])
def test_numbers_that_no_row_sees_may_be_anything(maps, window, chunked, group, page, value):
    """Slots behind a request's last key hold what a former owner left; one token's key and value are not finite."""
    from atom_b200 import native

    q_lens, past, nkv, dk, column = [70, 1, 300], [30, 200, 5], 2, 128 // maps, 77
    nh, T = nkv * group, sum(q_lens)
    g = torch.Generator().manual_seed(7)
    bf = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16).to(DEV)  # noqa: E731
    q, gate = bf(T, nh * maps * dk), bf(T, nh)
    n_pages = [-(-(a + n) // page) for a, n in zip(past, q_lens)]
    table = torch.full((3, max(n_pages)), -1, dtype=torch.int32)
    at = 1
    for i, n in enumerate(n_pages):
        table[i, :n] = torch.arange(at, at + n)
        at += n
    kp, vp = bf(at + 1, nkv * maps, page, dk), bf(at + 1, nkv, page, 128)
    cu, ctx = _arrays(q_lens, past)

    def run():
        out = torch.empty((T, nh * 128), dtype=torch.bfloat16, device=DEV)
        native.window_prefill(out, q, kp, vp, table.to(DEV), cu, ctx, 3, nh, nkv, dk, dk ** -0.5, window, None, gate, 1.0, chunked,
                              (0.4, 1e-5) if maps == 2 else None)
        native.check_error_flags()
        return out.view(T, nh, 128)

    def spoil():
        for i, n in enumerate(n_pages):
            last, behind = int(table[i, n - 1]), (past[i] + q_lens[i] - 1) % page + 1
            kp[last, :, behind:] = vp[last, :, behind:] = value
        kp[0], vp[0], kp[at], vp[at] = value, value, value, value
        seen = [past[0] + 33, -1, -1]
        page_of = int(table[0, seen[0] // page])
        vp[page_of, :, seen[0] % page, column] = value
        return seen

    if maps == 2:                                     # (a value that is not finite reaches the row's mean square: all columns)
        column = slice(None)
    _same_where_unseen(run, spoil, q_lens, past, window, chunked, column)


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("shared,window", [(64, 0), (64, 150), (0, 100)])
def test_requests_beside_one_another_in_arrays(shared, window, value):
    """Tiles of keys reach into the rows of the requests before and behind: one of these has numbers that are not finite."""
    from atom_b200 import native

    q_lens, past, heads = [60, 129, 40], [10, 300, 0], 3
    T = sum(q_lens)
    g = torch.Generator().manual_seed(9)
    bf = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16).to(DEV)  # noqa: E731
    first = [max(0, a - window + 1) if window else 0 for a in past]
    keys = [a + n - f for a, n, f in zip(past, q_lens, first)]
    q, k, v, extra = bf(T, heads, 128 + shared), bf(sum(keys), heads * 128), bf(sum(keys), heads * 128), bf(sum(keys), 64)
    cu, ctx = _arrays(q_lens, past)

    def run():
        out = torch.empty((T, heads, 128), dtype=torch.bfloat16, device=DEV)
        native.dense_prefill(out, q, k, v, extra if shared else None, cu, ctx, 3, 0.09, window)
        native.check_error_flags()
        return out

    def spoil():
        key = past[1] + 100
        v[keys[0] + key - first[1]] = value
        k[keys[0] + key - first[1], 3] = value
        return [-1, key, -1]

    _same_where_unseen(run, spoil, q_lens, past, window, False, slice(None))


@pytest.mark.parametrize("maps", [1, 2])
@pytest.mark.parametrize("q_lens", [[1 + i % 3 for i in range(700)], [0, 5, 0] + [1 + 7 * i % 190 for i in range(60)], [33] * 9], ids=["700", "60", "9"])
def test_every_unit_is_taken_once(q_lens, maps):
    """More units than threads that sort them, many of equal lengths, requests without rows: every row is the plain kernel's (its
    bound and the roundings of two outputs)."""
    from atom_b200 import native

    nkv, group, page, dk, scale = 2, 8, 8, 128 // maps, 0.1
    nh, T, past = nkv * group, sum(q_lens), [(37 * i) % 300 for i in range(len(q_lens))]
    g = torch.Generator(device=DEV).manual_seed(maps)
    bf = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)  # noqa: E731
    need = [-(-(a + n) // page) for a, n in zip(past, q_lens)]
    table = torch.full((len(q_lens), max(need)), -1, dtype=torch.int32)
    at = 0
    for i, n in enumerate(need):
        table[i, :n] = torch.arange(at, at + n)
        at += n
    q, kp, vp, table = bf(T, nh * maps * dk), bf(at, nkv * maps, page, dk), bf(at, nkv, page, 128), table.to(DEV)
    cu, ctx = _arrays(q_lens, past)
    pos = torch.cat([torch.arange(a, a + n) for a, n in zip(past, q_lens)]).to(torch.int32).to(DEV)
    sot = torch.cat([torch.full((n,), i) for i, n in enumerate(q_lens)]).to(torch.int32).to(DEV)
    got, want = (torch.full((T, nh * 128), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(2))
    two = (0.4, 1e-5) if maps == 2 else None
    native.window_prefill(got, q, kp, vp, table, cu, ctx, len(q_lens), nh, nkv, dk, scale, 100, maps=two)
    native.window_attention(want, q, kp, vp, table, pos, sot, nh, nkv, dk, 128, scale, window=100, maps=two)
    native.check_error_flags()
    assert _rel(got, want.double().cpu()) <= 5e-3


@pytest.mark.parametrize("dk,H,G,GV,dv", [(64, 32, 8, 4, 128), (64, 3, 1, 2, 8), (128, 5, 0, 0, 64), (256, 2, 2, 2, 72), (64, 1, 1, 1, 16)])
@pytest.mark.parametrize("norm", [None, torch.bfloat16, torch.float32], ids=str)
@pytest.mark.parametrize("T", [1, 37])
def test_rows_rotated_whole(T, norm, dk, H, G, GV, dv):
    """Queries, keys and values of rows whose heads are rotated from end to end, against 64-bit; a padding row and a token without a page."""
    from atom_b200 import native

    g = torch.Generator(device=DEV).manual_seed(dk + H)
    bf = lambda *s: torch.randn(s, generator=g, device=DEV).to(torch.bfloat16)  # noqa: E731
    C, page, mag = (H + G) * dk + GV * dv, 16, 1.25
    qkv = bf(T, C + 8)[:, :C]
    freq = torch.rand(dk // 2, generator=g, device=DEV)
    w = [(torch.rand(dk, generator=g, device=DEV) + 0.5).to(norm) for _ in range(2)] if norm else None
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    pos, sot = torch.arange(T, dtype=torch.int32, device=DEV) + 5, torch.zeros(T, dtype=torch.int32, device=DEV)
    pages = -(-(T + 5) // page)
    bt, status = i32([list(range(pages))]), torch.zeros(1, dtype=torch.int32, device=DEV)
    kp, vp = bf(pages, max(G, 1), page, dk), bf(pages, max(GV, 1), page, dv)
    q = torch.full((T, H * dk), float("nan"), dtype=torch.bfloat16, device=DEV)
    if T > 1:
        sot[T - 1] = -1
    keep = kp.clone()
    torch.cuda.synchronize()      # (kernels made the index arrays)
    native.conv_rope_write(q, qkv, H, G, dk, dv, None, None, freq, dk, pos, sot, i32([0, T]), i32([0]), bt, page, kp if G else None,
                           vp if G else None, status, magnitude=mag, value_heads=GV, head_norms=(w[0], w[1], 1e-5) if norm else None)
    x = qkv.double()[:, : (H + G) * dk].unflatten(1, (H + G, dk))
    if norm:
        x = x / (x.square().mean(-1, keepdim=True) + 1e-5).sqrt() * torch.cat([w[0].expand(H, dk), w[1].expand(G, dk)]).double()
    a = (pos.double()[:, None] * freq.double())[:, None]
    x1, x2 = x[..., : dk // 2], x[..., dk // 2:]
    want = torch.cat([x1 * a.cos() - x2 * a.sin(), x2 * a.cos() + x1 * a.sin()], -1) * mag
    n = T - 1 if T > 1 else T
    assert _rel(q[:n].view(n, H, dk), want[:n, :H].cpu()) <= 2.5e-3 and bool(q[n:].isnan().all())
    if G:
        at = lambda p, i: p[(i + 5) // page, :, (i + 5) % page]  # noqa: E731
        assert _rel(torch.stack([at(kp, i) for i in range(n)]), want[:n, H:].cpu()) <= 2.5e-3
        assert torch.equal(torch.stack([at(vp, i) for i in range(n)]), qkv[:n, (H + G) * dk:].unflatten(1, (GV, dv)))
        assert torch.equal(kp[:, :, :][0, :, :5], keep[0, :, :5]) and not int(status)
        native.conv_rope_write(q, qkv, H, G, dk, dv, None, None, freq, dk, pos, sot, i32([0, T]), i32([0]), i32([[-1] * pages]), page, kp, vp,
                               status, value_heads=GV, head_norms=(w[0], w[1], 1e-5) if norm else None)
        assert int(status) == 1
