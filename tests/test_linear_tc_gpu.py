"""The recurrences with a matrix state in chunks on the tensor cores (csrc/linear_attention_tc.cu) against the recurrence
row by row in 64-bit over the same inputs: sizes at the edges of chunks, blocks and tiles, requests that continue, mild and
sudden decays."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
F64 = torch.float64
LENS = [[65], [1, 200, 16, 63], [64, 129], [15, 17, 1, 1, 80]]
SIZES = [(128, 128), (64, 64), (40, 72), (8, 8)]


def _case(lens, dk, dv, H, decay, seed):
    g = torch.Generator().manual_seed(seed)
    T, n = sum(lens), len(lens)
    rand = lambda *s: torch.randn(*s, generator=g, dtype=F64)  # noqa: E731
    slots = torch.randperm(n + 2, generator=g)[:n]
    x = rand(T, 2 * H * dk + 2 * H * dv).to(torch.bfloat16)
    # what the decays are formed from: most channels forget little; "sudden": some rows forget nearly everything
    z = rand(T, H * dk).float()
    if decay == "sudden":
        z = torch.where(torch.rand(T, H * dk, generator=g) < 0.2, torch.full_like(z, 30.0), z)
    return T, n, slots, x, z, rand(n + 2, H, dk, dv).float()


def _walk(q, k, v, log_a, S, lens, slots, before=False, u=None):
    """Row by row in 64-bit: outputs [T, H, dv] and the states after."""
    o, S, at = torch.empty_like(v), S.double().clone(), 0
    for n, slot in zip(lens, slots.tolist()):
        s = S[slot]
        for t in range(at, at + n):
            kv = k[t][:, :, None] * v[t][:, None, :]
            if before:
                o[t] = torch.einsum("hk,hkv->hv", q[t], s + u[:, :, None] * kv)
            s = torch.exp(log_a[t])[:, :, None] * s + kv
            if not before:
                o[t] = torch.einsum("hk,hkv->hv", q[t], s)
        S[slot] = s
        at += n
    return o, S


def _rel(got, want):
    return float((got.double().cpu() - want).norm() / want.norm())


def _arrays(lens, slots):
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).to(torch.int32)
    return cu.to(DEV), slots.to(torch.int32).to(DEV)


def _lightning(lens, dk, dv, decay, seed, write_state=True):
    from atom_b200 import native

    H = 3
    T, n, slots, x, _, S = _case(lens, dk, dv, H, decay, seed)
    lam = torch.tensor([0.99, 0.6, 0.0 if decay == "sudden" else 0.9])
    act = torch.nn.functional.silu(x.double())
    q, k, v = (t.unflatten(1, (H, -1)) for t in act[:, : 2 * H * dk + H * dv].split([H * dk, H * dk, H * dv], 1))
    want = _walk(q, k, v, torch.log(lam.double())[None, :, None].expand(T, H, dk), S, lens, slots)
    cu, sl = _arrays(lens, slots)
    out, state = torch.empty(T, H * dv, device=DEV), S.to(DEV)
    scratch = torch.empty(native.lightning_scratch_elems(T, n, H, dk, dv), device=DEV)
    native.lightning_scan(out, x.to(DEV), lam.to(DEV), state, scratch, cu, sl, n, H, dk, dv, write_state)
    return out.unflatten(1, (H, dv)), state, want


def _gla(lens, dk, dv, decay, seed, write_state=True):
    from atom_b200 import native

    H, tau, scale = 2, 4.0, dk ** -0.5
    T, n, slots, x, z, S = _case(lens, dk, dv, H, decay, seed)
    z = -z if decay == "sudden" else z + 1.0
    z = z * (40.0 if decay == "sudden" else 1.0)
    bias = torch.linspace(-1, 3, H * dk).to(torch.bfloat16)
    q, k, v = (t.unflatten(1, (H, -1)) for t in x[:, : 2 * H * dk + H * dv].double().split([H * dk, H * dk, H * dv], 1))
    log_a = torch.nn.functional.logsigmoid(z.double() + bias.double()).unflatten(1, (H, dk)) / tau
    want = _walk(q * scale, k, v, log_a, S, lens, slots)
    cu, sl = _arrays(lens, slots)
    xd, out, state = x.to(DEV), torch.empty(T, H * dv, device=DEV), S.to(DEV)
    nb, na = native.gla_scratch_elems(T, n, H, dk, dv)
    sb, sa = torch.empty(nb, device=DEV), torch.empty(na, device=DEV)
    native.gla_scan(out, xd[:, : H * dk], xd[:, H * dk:2 * H * dk], xd[:, 2 * H * dk:2 * H * dk + H * dv], z.to(DEV), bias.to(DEV),
                    tau, scale, state, sb, sa, cu, sl, n, H, dk, dv, write_state)
    return out.unflatten(1, (H, dv)), state, want


def _wkv(lens, dk, dv, decay, seed, write_state=True):
    from atom_b200 import native

    H, eps = 2, 1e-5
    T, n, slots, x, z, S = _case(lens, dk, dv, H, decay, seed)
    w0 = torch.linspace(-5, 1, H * dk).to(torch.bfloat16)
    u, nw = torch.linspace(-1, 1, H * dk).to(torch.bfloat16), torch.linspace(0.5, 1.5, H * dv).to(torch.bfloat16)
    r, k, v, gate = (t.contiguous() for t in x.split([H * dk, H * dk, H * dv, H * dv], 1))
    heads = lambda t: t.double().unflatten(1, (H, -1))  # noqa: E731
    o, Sw = _walk(heads(r), heads(k), heads(v), -torch.exp((z.double() + w0.double()).clamp(max=20)).unflatten(1, (H, dk)), S, lens,
                  slots, True, u.double().view(H, dk))
    o = o / (o.square().mean(-1, keepdim=True) + eps).sqrt() * nw.double().view(H, dv)
    cu, sl = _arrays(lens, slots)
    y, state = torch.empty(T, H * dv, dtype=torch.bfloat16, device=DEV), S.to(DEV)
    scratch = torch.empty(max(1, native.wkv_scratch_elems(T, n, H, dk, dv)), device=DEV)
    d = lambda t: t.to(DEV)  # noqa: E731
    native.wkv(y, d(r), d(k), d(v), d(z), d(gate), d(w0), d(u), d(nw), state, cu, sl, n, H, dk, dv, eps, write_state, scratch)
    return y.unflatten(1, (H, dv)), state, (o * torch.nn.functional.silu(heads(gate)), Sw)


KINDS = {"lightning": _lightning, "gla": _gla, "wkv": _wkv}


@pytest.mark.parametrize("decay", ["mild", "sudden"])
@pytest.mark.parametrize("dk,dv", SIZES)
@pytest.mark.parametrize("lens", LENS, ids=str)
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_chunks_against_the_recurrence_in_64_bits(kind, lens, dk, dv, decay):
    """32-bit operands enter the products with all their bits and the sums are 32-bit: an error of some 2^-24 for every
    product and sum on the way, 3e-6 with room for the decays' exponentials (two units in the last place each); the rows
    of "wkv" are rounded to bfloat16 (2^-9)."""
    from atom_b200 import native

    if kind == "wkv" and dv > 64:
        pytest.skip("runs row by row")
    assert native.linear_tc_elems(sum(lens), len(lens), 2, dk, dv, True)[0]
    out, state, (want, want_state) = KINDS[kind](lens, dk, dv, decay, seed=len(lens) + dk)
    assert _rel(out, want) <= (3e-3 if kind == "wkv" else 3e-6)
    assert _rel(state, want_state) <= 3e-6


@pytest.mark.parametrize("dk,dv", [(128, 128), (64, 128), (40, 72), (128, 136)])
@pytest.mark.parametrize("kind", ["gla", "lightning"])
def test_value_columns_in_narrow_and_wide_tiles(kind, dk, dv, monkeypatch):
    """Steps of few chunks take their value columns in tiles of 64, others in tiles of 128: as near to 64-bit as the test above has
    it, and the same numbers for a request that is alone and for one with 120 more behind it."""
    many = [100] + [1, 2, 65] * 40
    T = sum(many)
    chunks = sum(-(-n // 64) for n in many)
    assert chunks * 2 > 148 and 2 * 3 * 2 <= 148
    wide, state, (want, want_state) = KINDS[kind](many, dk, dv, "mild", seed=3)
    assert wide.shape[0] == T and _rel(wide, want) <= 3e-6 and _rel(state, want_state) <= 3e-6
    case = _case

    def first(lens, dk, dv, H, decay, seed):
        _, _, slots, x, z, S = case(many, dk, dv, H, decay, seed)
        return 100, 1, slots[:1], x[:100], z[:100], S

    monkeypatch.setitem(globals(), "_case", first)
    narrow, _, _ = KINDS[kind]([100], dk, dv, "mild", seed=3)
    assert torch.equal(narrow, wide[:100])


@pytest.mark.parametrize("kind", sorted(KINDS))
def test_state_is_left_alone_where_it_is_not_written(kind):
    out, state, (want, _) = KINDS[kind]([70, 3], 64, 64, "mild", seed=5, write_state=False)
    assert _rel(out, want) <= (3e-3 if kind == "wkv" else 3e-6)
    assert torch.equal(state.cpu(), _case([70, 3], 64, 64, 3 if kind == "lightning" else 2, "mild", 5)[5])


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("which", ["key", "value"])
@pytest.mark.parametrize("dk,dv", [(128, 128), (64, 64), (40, 64)])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_a_row_that_is_not_finite_reaches_no_earlier_row(kind, dk, dv, which, value, monkeypatch):
    """One number of one row: the rows before it and the other requests keep what the walk row by row gives them (the bounds
    of both), the request's rows from there on show it."""
    from atom_b200 import native

    if kind == "wkv" and dv > 64:
        pytest.skip("runs row by row")
    lens, bad = [5, 100, 70], 5 + 64 + 21           # in the second chunk of the second request, inside a block of 16 rows
    H = 3 if kind == "lightning" else 2
    real = _case

    def spoilt(*args):
        T, n, slots, x, z, S = real(*args)
        x[bad, H * dk + 3 if which == "key" else 2 * H * dk + 3] = value
        return T, n, slots, x, z, S

    monkeypatch.setitem(globals(), "_case", spoilt)
    out, state, _ = KINDS[kind](lens, dk, dv, "mild", seed=3)
    monkeypatch.setattr(native, "LINEAR_TC", False)
    want, want_state, _ = KINDS[kind](lens, dk, dv, "mild", seed=3)
    assert torch.equal(torch.isfinite(out), torch.isfinite(want)) and not bool(torch.isfinite(out[bad:105]).all())
    assert torch.equal(torch.isfinite(state), torch.isfinite(want_state))
    keep = torch.ones(len(out), dtype=torch.bool)
    keep[bad:105] = False
    assert bool(torch.isfinite(out[keep]).all())
    assert _rel(out[keep], want[keep].double().cpu()) <= (4e-3 if kind == "wkv" else 3e-6)


@pytest.mark.parametrize("ns,n", [(96, 0), (300, 0), (128, 40), (128, 256)])
def test_many_single_rows_are_walked(ns, n):
    """Steps of the decayed recurrence whose chunks would hold a row each are left to the walk; as many rows of one request are not."""
    from atom_b200 import native

    T, S, H, dk = ns + n, ns + (n > 0), 32, 64
    assert native.wkv_scratch_elems(T, S, H, dk, dk, max(n, 1)) == 0
    assert n or native.wkv_scratch_elems(T, S, H, dk, dk) == 0
    assert native.wkv_scratch_elems(T, 1, H, dk, dk, T) > 0


@pytest.mark.parametrize("lens", [[100], [3, 64, 80]], ids=str)
@pytest.mark.parametrize("kind", ["gla", "wkv"])
def test_what_is_forgotten_at_once_leaves_nothing(kind, lens, monkeypatch):
    """Some rows forget everything in some channels: of a state of 2^60 nothing is left there, as in 64-bit (the bounds above)."""
    real = _case

    def forgetful(lens_, dk, dv, H, decay, seed):
        T, n, slots, x, z, S = real(lens_, dk, dv, H, "mild", seed)
        rows = torch.zeros(T, dtype=torch.bool)
        rows[[0] + torch.tensor(lens_).cumsum(0)[:-1].tolist() + [T - 9]] = True
        z[rows] = 1e4 if kind == "wkv" else -1e4
        return T, n, slots, x, z, S * 2.0 ** 60

    monkeypatch.setitem(globals(), "_case", forgetful)
    out, state, (want, want_state) = KINDS[kind](lens, 64, 64, "mild", seed=4)
    T = sum(lens)
    first = torch.tensor([0] + torch.tensor(lens).cumsum(0)[:-1].tolist())
    after = torch.ones(T, dtype=torch.bool)
    after[first] = kind != "wkv"                     # (the decayed recurrence's row sees the state before it forgets)
    assert _rel(out[after], want[after]) <= (3e-3 if kind == "wkv" else 3e-6)
    used = want_state.abs().amax((1, 2, 3)) < 2.0 ** 30
    assert int(used.sum()) == len(lens) and _rel(state[used], want_state[used]) <= 3e-6


@pytest.mark.parametrize("dk,dv", [(128, 128), (64, 64)])
def test_lightning_chunks_are_as_near_as_the_walk(dk, dv):
    """Operands' roundings (silu, 2^-24 each) are what is left: 0.7 to 0.9e-7 with either, and 1.1e-7 with room for other numbers;
    states, sums over a thousand rows, 1.3e-7 walked and less in chunks."""
    for seed in (1, 2):
        out, state, (want, want_state) = _lightning([700, 64, 300], dk, dv, "mild", seed)
        assert _rel(out, want) <= 1.1e-7 and _rel(state, want_state) <= 1.25e-7
