"""Attention of prompt portions with mixed heads on tcgen05 (csrc/attention_mixed_prefill.cu) against 64-bit: 1, 2 and 4 key heads,
with and without distance bias, sink, temperature and window, requests at the edges of tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
F64 = torch.float64


@pytest.mark.parametrize("q_lens,past", [([40], [0]), ([1, 130, 3, 257], [700, 0, 64, 31]), ([500, 1, 33], [1000, 127, 128]),
                                         ([64, 7, 0, 90], [8300, 40, 5, 9000]), ([1 + i % 3 for i in range(330)], [(5 * i) % 40 for i in range(330)])],
                         ids=lambda v: str(v)[:40])
@pytest.mark.parametrize("nkv,page,window,extras", [(4, 16, 0, True), (2, 8, 300, True), (1, 128, 0, True), (4, 64, 1, False), (2, 16, 0, False)])
def test_portions(q_lens, past, nkv, page, window, extras):
    """Outputs are rounded to bfloat16 (2^-9); mixed queries keep 17 bits, weights 16."""
    from atom_b200 import native
    from atom_b200.parts.mixed_attention import distance_thresholds

    nh, T, scale, coef, every = 4 * nkv, sum(q_lens), 0.1, 0.5, 64
    g = torch.Generator().manual_seed(nkv + window)
    rand = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    bf = lambda *s: rand(*s).to(torch.bfloat16)  # noqa: E731
    q, talk = bf(T, nh * 128 + 64), torch.eye(nh) + 0.2 * rand(nh, nh)
    rel, sink = (rand(32, nh), rand(nh) * 2) if extras else (None, None)
    thr = distance_thresholds(32, 4096)
    n_pages = [-(-(a + n) // page) for a, n in zip(past, q_lens)]
    perm = torch.randperm(sum(n_pages) + 2, generator=g).tolist()
    table = torch.full((len(q_lens), max(n_pages)), -1, dtype=torch.int32)
    kp, vp = bf(len(perm), nkv, page, 128), bf(len(perm), nkv, page, 128)
    want, at = torch.empty(T, nh, 128, dtype=F64), 0
    for i, (a, n) in enumerate(zip(past, q_lens)):
        table[i, : n_pages[i]] = torch.tensor([perm.pop() for _ in range(n_pages[i])], dtype=torch.int32)
        rows = table[i, : n_pages[i]].long()
        k = kp[rows].double().transpose(1, 2).reshape(-1, nkv, 128)[: a + n]
        v = vp[rows].double().transpose(1, 2).reshape(-1, nkv, 128)[: a + n]
        dist = torch.arange(a, a + n)[:, None] - torch.arange(a + n)[None]
        ok = dist >= 0
        if window:
            ok &= dist < window
        bucket = torch.where(dist < 16, dist.clamp(min=0), 16 + sum((dist >= t).long() for t in thr))
        temp = 1 + coef * torch.log(torch.floor((torch.arange(a, a + n).double() + 1) / every) + 1) if extras else torch.ones(n, dtype=F64)
        qq = q[at:at + n, : nh * 128].double().view(n, nh, 128)
        s = torch.stack([qq[:, h] @ k[:, h // 4].T * (scale * temp)[:, None] + (rel[:, h].double()[bucket] if extras else 0) for h in range(nh)])
        for h in range(nh):
            m = torch.einsum("g,gij->ij", talk[h].double(), s).masked_fill(~ok, float("-inf"))
            if extras:
                m = torch.cat([m, sink[h].double().expand(n, 1)], 1)
            want[at:at + n, h] = m.softmax(1)[:, : a + n] @ v[:, h // 4]
        table[i, : int(ok.any(0).float().argmax()) // page] = -1       # pages that no row of the step sees have been given back
        at += n
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    d = lambda t: t.to(DEV) if t is not None else None  # noqa: E731
    cu, ctx = i32([0] + torch.tensor(q_lens).cumsum(0).tolist()), i32([a + n for a, n in zip(past, q_lens)])
    out = torch.full((T, nh * 128), float("nan"), dtype=torch.bfloat16, device=DEV)
    assert native.attention_mixed_prefill_supports(nh, nkv, 128, 128, page, 32, len(thr))
    native.attention_mixed_prefill(out, d(q), d(kp), d(vp), d(table), cu, ctx, len(q_lens), nh, nkv, scale, window, d(rel), 16 if extras else 0,
                                   i32(thr) if extras else None, d(talk), d(sink), coef if extras else 0.0, every if extras else 0)
    native.check_error_flags()
    assert float((out.double().cpu().view(T, nh, 128) - want).norm() / want.norm()) <= 3e-3


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("nkv,page,window", [(4, 16, 0), (2, 64, 100), (1, 16, 0)])
def test_numbers_that_no_row_sees_may_be_anything(nkv, page, window, value):
    """Slots behind a request's last key hold what a former owner left; one token's key and value are not finite.  Rows that see
    none of it keep their results (up to one more rounding to bfloat16 on either side: 2^-7 of a number)."""
    from atom_b200 import native
    from atom_b200.parts.mixed_attention import distance_thresholds

    q_lens, past, nh = [70, 1, 100], [30, 200, 5], 4 * nkv
    T, spoilt = sum(q_lens), 30 + 33
    g = torch.Generator().manual_seed(nkv)
    rand = lambda *s: torch.randn(*s, generator=g).to(DEV)  # noqa: E731
    bf = lambda *s: rand(*s).to(torch.bfloat16)  # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    q, talk, rel, sink, thr = bf(T, nh * 128), torch.eye(nh, device=DEV) + 0.2 * rand(nh, nh), rand(32, nh), rand(nh), i32(distance_thresholds(32, 4096))
    n_pages = [-(-(a + n) // page) for a, n in zip(past, q_lens)]
    table = torch.full((3, max(n_pages)), -1, dtype=torch.int32)
    at = 0
    for i, n in enumerate(n_pages):
        table[i, :n] = torch.arange(at, at + n)
        at += n
    kp, vp = bf(at, nkv, page, 128), bf(at, nkv, page, 128)
    cu, ctx = i32([0] + torch.tensor(q_lens).cumsum(0).tolist()), i32([a + n for a, n in zip(past, q_lens)])

    def run():
        out = torch.empty((T, nh * 128), dtype=torch.bfloat16, device=DEV)
        native.attention_mixed_prefill(out, q, kp, vp, table.to(DEV), cu, ctx, 3, nh, nkv, 0.05, window, rel, 16, thr, talk, sink, 0.5, 64)
        native.check_error_flags()
        return out.float().cpu()

    clean = run()
    for i, n in enumerate(n_pages):
        behind = (past[i] + q_lens[i] - 1) % page + 1
        kp[int(table[i, n - 1]), :, behind:] = vp[int(table[i, n - 1]), :, behind:] = value
    kp[int(table[0, spoilt // page]), 0, spoilt % page, 5] = value
    vp[int(table[0, spoilt // page]), :, spoilt % page] = value
    got = run()
    pos = torch.cat([torch.arange(a, a + n) for a, n in zip(past, q_lens)])
    sees = (pos >= spoilt) & (torch.arange(T) < q_lens[0]) & ((pos - spoilt < window) if window else torch.ones(T, dtype=torch.bool))
    assert not bool(torch.isfinite(got[sees]).any())
    torch.testing.assert_close(got[~sees], clean[~sees], rtol=2 ** -7, atol=2e-3)
