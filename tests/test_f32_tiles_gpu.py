"""32-bit products and attention in tiles: every tile size of the products at its edges, the products of many rows on the
tensor cores (three numbers for one) with numbers that are not finite among them, and the attention's two tile sizes over
ragged requests, against 64-bit."""
import pytest
import torch

from test_kernels_gpu import _paged_case, _ref_attention

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _rand(shape, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


def _rel(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 32, 33, 48, 49, 256, 257])
@pytest.mark.parametrize("N,K", [(31, 4), (64, 100), (2500, 516)])
def test_product_in_tiles_on_the_fma_units(M, N, K):
    """Two sequential sums of K / 2 terms, each with an error of some 2^-24 of a partial sum: about sqrt(K) 2^-24 relative."""
    from atom_b200 import native

    a, w, bias = _rand((M, K + 4), 1)[:, :K], _rand((N, K), 2), _rand((N,), 3)
    out = torch.empty((M, N), device=DEV)
    native.gemm_f32(out, a, w, bias)
    assert _rel(out, a.double() @ w.double().T + bias.double()) <= 2e-6


@pytest.mark.parametrize("M,N,K", [(160, 128, 64), (161, 130, 100), (300, 2050, 516), (700, 1000, 66), (1030, 4100, 4096)])
def test_product_of_many_rows_on_the_tensor_cores(M, N, K, monkeypatch):
    """No further from 64-bit than the FMA units' sums over the same numbers, with room for a few units in the last place."""
    from atom_b200 import native

    monkeypatch.setattr(native, "F32_TC_MIN_PRODUCTS", 0)
    a, w, bias = _rand((M, K), 4), _rand((N, K), 5), _rand((N,), 6)
    want = a.double() @ w.double().T + bias.double()
    out, fma = torch.empty((M, N + 3), device=DEV)[:, :N], torch.empty((M, N), device=DEV)
    native.gemm_f32(out, a, w, bias)
    monkeypatch.setattr(native, "F32_TC_MIN_ROWS", 0)
    native.gemm_f32(fma, a, w, bias)
    assert not torch.equal(out, fma)
    assert _rel(out, want) <= max(_rel(fma, want), 4e-7)
    native.check_error_flags()


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.4e38, 1e-36])
@pytest.mark.parametrize("where", ["a", "w"])
def test_product_of_many_rows_with_a_number_that_is_not_finite(value, where, monkeypatch):
    """Outputs of a row (of A or W) with a number that its three do not hold are the FMA units', bit for bit; the others are what
    they are without it."""
    from atom_b200 import native

    monkeypatch.setattr(native, "F32_TC_MIN_PRODUCTS", 0)
    a, w = _rand((200, 128), 7), _rand((300, 128), 8)
    clean, out, fma = (torch.empty((200, 300), device=DEV) for _ in range(3))
    native.gemm_f32(clean, a, w)
    (a if where == "a" else w)[17, 100] = value
    native.gemm_f32(out, a, w)
    monkeypatch.setattr(native, "F32_TC_MIN_ROWS", 0)
    native.gemm_f32(fma, a, w)
    if where == "a":
        clean[17] = fma[17]
    else:
        clean[:, 17] = fma[:, 17]
    assert torch.equal(out.view(torch.int32), clean.view(torch.int32))


@pytest.mark.parametrize("N,K", [(700, 1000), (130, 66), (1030, 4096)])
def test_a_row_of_a_product_does_not_depend_on_the_others(N, K, monkeypatch):
    """Bit for bit, over every width of the tensor cores' tiles, at their edges."""
    from atom_b200 import native

    for least in (0, 1 << 40):              # on the tensor cores, on the FMA units
        monkeypatch.setattr(native, "F32_TC_MIN_PRODUCTS", least)
        a, w = _rand((400, K), 1), _rand((N, K), 2)
        whole = torch.empty((400, N), device=DEV)
        native.gemm_f32(whole, a, w)
        for M in (1, 15, 16, 17, 32, 33, 64, 65, 127, 130, 399):
            for at in (0, 400 - M):
                out = torch.empty((M, N), device=DEV)
                native.gemm_f32(out, a[at:at + M], w)
                assert torch.equal(out, whole[at:at + M]), (M, at)
    native.check_error_flags()


@pytest.mark.parametrize("K", [260, 512, 1000, 1001, 1024, 1028])
@pytest.mark.parametrize("M", [5, 64, 300])
def test_a_column_of_a_product_does_not_depend_on_the_others(M, K):
    """Bit for bit: an output's sums are cut alike however tall W is, and however W's rows are brought (K 1,001)."""
    from atom_b200 import native

    a, w = _rand((M, K), 1), _rand((20480, K), 2)
    whole, part = torch.empty((M, 20480), device=DEV), torch.empty((M, 4224), device=DEV)
    native.gemm_f32(whole, a, w)
    native.gemm_f32(part, a, w[:4224])
    assert torch.equal(whole[:, :4224], part)
    native.check_error_flags()


@pytest.mark.parametrize("K,N", [(40, None), (64, None), (130, None), (256, 6200), (259, 6200), (1000, 8500), (1024, 8400), (1100, 4200),
                                 (1100, 6200), (2056, 8500)])
def test_quarters_of_k_in_one_cta_or_four(K, N):
    """Bit for bit: enough rows that a CTA takes all of K, and few, where four take a quarter each, some of them empty or ragged, and
    matrices whose K is never cut; with a bias, and no further from 64-bit than sums of K / 4 and of 4 in 32-bit are."""
    from atom_b200 import native

    N = N or -(-(1 << 20) // K)
    a, w, bias = _rand((1300 if K >= 256 else 150, K), 1), _rand((N, K), 2), _rand((N,), 3)
    whole = torch.empty((a.shape[0], N), device=DEV)
    native.gemm_f32(whole, a, w, bias)
    assert _rel(whole, a.double() @ w.double().T + bias.double()) <= 4e-7
    for M in (1, 16, 17, 33, 64, 65, 129):
        out = torch.empty((M, N), device=DEV)
        native.gemm_f32(out, a[-M:], w, bias)
        assert torch.equal(out, whole[-M:]), M
    native.check_error_flags()


@pytest.mark.parametrize("a_off,w_off", [(1, 0), (0, 1), (3, 2)])
@pytest.mark.parametrize("K,N", [(1024, 1100), (1028, 4200), (2052, 700), (28, 40000)])
def test_rows_that_begin_anywhere(K, N, a_off, w_off):
    """The same bits wherever the rows of A and of W begin, and with A's rows further apart than K."""
    from atom_b200 import native

    def at(x, off, ld):
        buf = torch.full((x.shape[0] * ld + off,), float("nan"), device=DEV)
        view = buf[off:].view(-1, ld)[:, : x.shape[1]]
        return view.copy_(x)

    a, w = _rand((300, K), 1), _rand((N, K), 2)
    for M in (1, 17, 64, 65, 300):
        want, out = torch.empty((M, N), device=DEV), torch.empty((M, N), device=DEV)
        native.gemm_f32(want, a[:M], w)
        native.gemm_f32(out, at(a[:M], a_off, K + a_off), at(w, w_off, K))
        torch.cuda.synchronize()
        assert torch.equal(out, want), M
    native.check_error_flags()


@pytest.mark.parametrize("K", [100_000, 150_000])
def test_product_over_many_numbers(K):
    """No K is too large, also where A's planes of a tile of rows would not fit the scratch: the sums of 64 are added one after another,
    an error of some sqrt(K / 64) 2^-24."""
    from atom_b200 import native

    a, w = _rand((170, K), 1), _rand((140, K), 2)
    out = torch.empty((170, 140), device=DEV)
    native.gemm_f32(out, a, w)
    native.check_error_flags()
    assert _rel(out, a.double() @ w.double().T) <= 3e-6


def test_product_of_numbers_near_the_smallest():
    """Where the lowest bits of a number lie below bfloat16's smallest, no bit is lost all the same."""
    from atom_b200 import native

    a, w = _rand((200, 1024), 1) * 2.0 ** -118, _rand((1100, 1024), 2) * 2.0 ** 60
    out = torch.empty((200, 1100), device=DEV)
    native.gemm_f32(out, a, w)
    assert _rel(out, a.double() @ w.double().T) <= 2e-6


def test_product_in_a_thread_that_has_called_nothing():
    """A host thread without a context of its own yet."""
    import threading

    from atom_b200 import native

    a, w, out, want = _rand((300, 4096), 1), _rand((2048, 4096), 2), torch.empty((300, 2048), device=DEV), torch.empty((300, 2048), device=DEV)
    native.gemm_f32(want, a, w)
    failed = []

    def work():
        try:
            native.gemm_f32(out[:299], a[:299], w)       # (rows that no map of another call describes)
        except Exception as e:
            failed.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not failed and torch.equal(out[:299], want[:299])


def test_products_of_two_threads_on_one_stream():
    """Nothing is shared between calls."""
    import threading

    from atom_b200 import native

    a, w = [_rand((300, 4096), i) for i in range(2)], [_rand((2048, 4096), 5 + i) for i in range(2)]
    want = [torch.empty((300, 2048), device=DEV) for _ in range(2)]
    for i in range(2):
        native.gemm_f32(want[i], a[i], w[i])
    wrong = []

    def work(i):
        try:
            outs = [torch.empty((300, 2048), device=DEV) for _ in range(40)]
            for o in outs:
                native.gemm_f32(o, a[i], w[i])
            wrong.extend(i for o in outs if not torch.equal(o, want[i]))
        except Exception as e:
            wrong.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("nh,nkv,hd,page,window", [(8, 2, 128, 16, 0), (5, 5, 64, 8, 0), (6, 2, 72, 16, 50), (4, 4, 16, 16, 0), (10, 2, 96, 4, 0)])
@pytest.mark.parametrize("q_lens,ctx_lens", [([1, 40, 3, 1], [77, 120, 3, 64]), ([300, 17], [420, 17]), ([1] * 6, [65, 64, 63, 1, 200, 129])])
def test_attention_in_tiles(nh, nkv, hd, page, window, q_lens, ctx_lens, monkeypatch):
    """32-bit scores, weights and sums: the bound of the kernel for any size."""
    from atom_b200 import native

    q, kp, vp, bt, dense = _paged_case(q_lens, ctx_lens, nh, nkv, hd, page, torch.float32, seed=3)
    T, scale = sum(q_lens), hd ** -0.5
    want = _ref_attention(q, dense, q_lens, ctx_lens, nh, nkv, scale, window)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    cu = i32([0] + torch.tensor(q_lens).cumsum(0).tolist())
    pos = i32([p for n, c in zip(q_lens, ctx_lens) for p in range(c - n, c)])
    sot = i32([s for s, n in enumerate(q_lens) for _ in range(n)])
    for sms in (1, 1 << 20):                # tiles of 64 rows, tiles of 16
        monkeypatch.setattr(native, "SM_COUNT", sms)
        out = torch.full((T, nh * hd), float("nan"), device=DEV)
        native.paged_attention_generic(out, q.reshape(T, nh * hd).contiguous().to(DEV), nh * hd, kp.to(DEV), vp.to(DEV),
                                       bt.contiguous().to(DEV), pos, sot, T, nh, nkv, hd, scale, window, cu, i32(ctx_lens), len(q_lens))
        torch.testing.assert_close(out.cpu().view(T, nh, hd), want, rtol=0, atol=2e-5)


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("nh,nkv,hd,window", [(8, 2, 128, 0), (6, 2, 72, 50), (5, 5, 64, 20)])
def test_attention_in_tiles_with_a_token_that_is_not_finite(nh, nkv, hd, window, value, monkeypatch):
    """Rows that do not see it keep what a block per token and head gives them (the two kernels' bound), the others show it."""
    from atom_b200 import native

    q_lens, ctx_lens, page, spoilt = [90, 1, 40], [100, 30, 200], 16, 37
    q, kp, vp, bt, _ = _paged_case(q_lens, ctx_lens, nh, nkv, hd, page, torch.float32, seed=5)
    vp[int(bt[0, spoilt // page]), :, spoilt % page] = value
    T = sum(q_lens)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    cu = i32([0] + torch.tensor(q_lens).cumsum(0).tolist())
    pos = i32([p for n, c in zip(q_lens, ctx_lens) for p in range(c - n, c)])
    sot = i32([s for s, n in enumerate(q_lens) for _ in range(n)])
    qd, kd, vd, bd = q.reshape(T, nh * hd).contiguous().to(DEV), kp.to(DEV), vp.to(DEV), bt.contiguous().to(DEV)

    def run():
        out = torch.empty((T, nh * hd), device=DEV)
        native.paged_attention_generic(out, qd, nh * hd, kd, vd, bd, pos, sot, T, nh, nkv, hd, hd ** -0.5, window, cu, i32(ctx_lens), len(q_lens))
        return out

    monkeypatch.setattr(native, "F32_TILES", False)
    want = run()
    monkeypatch.setattr(native, "F32_TILES", True)
    sees = (sot == 0) & (pos >= spoilt) & ((pos - spoilt < window) if window else torch.ones_like(pos, dtype=torch.bool))
    for sms in (1, 1 << 20):                # tiles of 64 rows, tiles of 16
        monkeypatch.setattr(native, "SM_COUNT", sms)
        got = run()
        assert bool(torch.isfinite(want[~sees]).all()) and not bool(torch.isfinite(got[sees]).any())
        torch.testing.assert_close(got[~sees], want[~sees], rtol=0, atol=2e-5)
