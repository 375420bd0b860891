"""The recurrence in chunks of tokens against the token-by-token sums in float64 and against the walk: every form of the decays,
requests around the length from which chunks are used and around whole chunks, decays of zero and below, decays that underflow,
heads that share q and k, column slices, slots that are not written, and rows that only the walk takes."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def plain(q, k, v, a, c, skip, S):
    """q, k [T, H, d], v [T, H, e], a [T, H, d or 1], c [T, H], S [H, d, e], all float64."""
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = a[t][:, :, None] * S + c[t][:, None, None] * k[t][:, :, None] * v[t][:, None, :]
        out[t] = torch.einsum("hde,hd->he", S, q[t]) + skip[:, None] * v[t]
    return out, S


def problem(form, heads, groups, vdim, lens, seed):
    g = torch.Generator().manual_seed(seed)
    T, d = sum(lens), 128
    p = dict(q=torch.randn(T, groups * d, generator=g), k=torch.randn(T, groups * d, generator=g), v=torch.randn(T, heads * vdim, generator=g),
             dt_dec=None, decay_head=None, decay_vec=None, skip=None)
    if form == "head":
        dec = torch.rand(heads, generator=g) * 0.5 + 0.5
        dec[0], dec[1 % heads] = 0.9995, -0.9
        p["decay_head"], a, c = dec, dec.expand(T, heads)[:, :, None], torch.ones(T, heads)
    elif form == "token":
        c, dec = torch.rand(T, heads, generator=g) * 2, torch.rand(T, heads, generator=g)
        dec[::37] = 0.0
        dec[50:60] = 1e-9
        p["dt_dec"], p["skip"], a = torch.cat([c, dec], 1), torch.randn(heads, generator=g), dec[:, :, None]
    else:
        f = torch.sigmoid(torch.randn(T, heads * d, generator=g) * 3) ** (1 / 16 if form == "channel" else 4)
        f[::41] = 0.0
        p["decay_vec"], a, c = f, f.view(T, heads, d), torch.ones(T, heads)
    state = torch.randn(len(lens) + 1, heads * vdim * d + 4, generator=g)
    ref, at = [], 0
    for i, n in enumerate(lens):
        r = slice(at, at + n)
        rep = lambda x: x[r].double().view(n, groups, d).repeat_interleave(heads // groups, 1)  # noqa: E731
        S = state[i, : heads * vdim * d].double().view(heads, vdim, d).transpose(1, 2)
        skip = p["skip"].double() if p["skip"] is not None else torch.zeros(heads, dtype=torch.float64)
        o, S = plain(rep(p["q"]), rep(p["k"]), p["v"][r].double().view(n, heads, vdim), a[r].double(), c[r].double(), skip, S)
        ref.append((o.reshape(n, -1), S.transpose(1, 2).reshape(-1)))
        at += n
    return p, state, ref


def run(p, state, lens, heads, groups, vdim, wide=4, write=True):
    from tokasaurus_b200.kernels import ops

    T = sum(lens)
    both = torch.zeros(T, p["q"].shape[1] * 2 + p["v"].shape[1] + wide)  # q, k and v as column slices of one tensor
    both[:, : p["q"].shape[1]], both[:, p["q"].shape[1]:2 * p["q"].shape[1]] = p["q"], p["k"]
    both[:, 2 * p["q"].shape[1]:both.shape[1] - wide] = p["v"]
    both = both.to(DEV)
    n = p["q"].shape[1]
    dev = lambda x: None if x is None else x.to(DEV)  # noqa: E731
    st, out = state.to(DEV), torch.full((T, heads * vdim), 7.0, device=DEV)
    starts = [sum(lens[:i]) for i in range(len(lens))]
    ops.decay_walk(both[:, :n], both[:, n:2 * n], both[:, 2 * n:both.shape[1] - wide], heads // groups, dev(p["dt_dec"]),
                   dev(p["decay_head"]), dev(p["skip"]), st, out, i32(list(range(len(lens)))), i32(starts), i32(lens), len(lens),
                   heads, 128, vdim, write, decay_vec=dev(p["decay_vec"]))
    return out.cpu(), st.cpu()


@pytest.mark.parametrize("form,heads,groups", [("head", 3, 3), ("token", 4, 2), ("channel", 2, 2), ("sharp", 2, 2)])
@pytest.mark.parametrize("vdim", [64, 128])
@pytest.mark.parametrize("lens", [[192], [191, 192, 193], [1, 256, 5, 257, 383], [40, 700]])
def test_chunks(form, heads, groups, vdim, lens, monkeypatch):
    from tokasaurus_b200.kernels import ops

    p, state, ref = problem(form, heads, groups, vdim, lens, 7 * sum(lens) + vdim)
    out, st = run(p, state, lens, heads, groups, vdim)
    monkeypatch.setattr(ops, "DECAY_CHUNKS_FROM", 1 << 30)
    walked, wst = run(p, state, lens, heads, groups, vdim)
    at, size = 0, heads * vdim * 128
    rel = lambda x, y: float((x.double() - y).norm() / y.norm())  # noqa: E731
    for i, n in enumerate(lens):
        o, S = ref[i]
        # a sum of some hundred float32 products, each exact to 2^-24 and rounded a few times on its way: 16 units in the last place
        assert rel(out[at:at + n], o) < 16 * 2.0 ** -24 and rel(st[i, :size], S) < 16 * 2.0 ** -24
        assert rel(out[at:at + n], o) < 1.5 * rel(walked[at:at + n], o) + 2.0 ** -24  # no less exact than the walk
        if n < 192:
            assert torch.equal(out[at:at + n], walked[at:at + n]) and torch.equal(st[i], wst[i])
        at += n
    assert torch.equal(st[:, size:], state[:, size:]) and torch.equal(st[-1], state[-1])  # nothing beside the requests' states
    monkeypatch.undo()
    again, kept = run(p, state, lens, heads, groups, vdim, write=False)
    assert torch.equal(again, out) and torch.equal(kept, state)
    odd, _ = run(p, state, lens, heads, groups, vdim, wide=3)  # strides that are no whole 16-byte pieces: the walk
    assert torch.equal(odd, walked)


def test_chunks_cut_into_steps():
    """A request in portions: chunks, walk, chunks, walk; the state goes from one to the other."""
    lens = [700]
    p, state, ref = problem("channel", 2, 2, 128, lens, 3)
    st, outs, at = state, [], 0
    for n in (200, 100, 321, 79):
        part = {k: (v[at:at + n] if v is not None and v.shape[0] == 700 else v) for k, v in p.items()}
        out, st = run(part, st, [n], 2, 2, 128)
        outs.append(out)
        at += n
    assert float((torch.cat(outs).double() - ref[0][0]).norm() / ref[0][0].norm()) < 16 * 2.0 ** -24


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("vdim,heads,lens", [(128, 2, [192, 1, 259]), (64, 3, [700, 191]), (128, 160, [200, 193])])
def test_chunks_of_the_forgetting_recurrence(dtype, vdim, heads, lens, monkeypatch):
    """S_t = diag(f) S + (1 - f) v^T with its gates and norm: chunks against the walk and float64; many heads too, for which the
    walk alone would not have split its gates from its sums."""
    from tokasaurus_b200.kernels import ops

    g = torch.Generator().manual_seed(heads)
    T, d = sum(lens), 128
    qfv = torch.randn(T, heads * (2 * d + vdim), generator=g)
    fb, low = torch.randn(heads * d, generator=g), torch.rand(heads * d, generator=g) * 0.95
    nw = torch.rand(vdim, generator=g) + 0.5
    state = torch.randn(len(lens) + 1, heads, vdim, d, generator=g)
    starts = [sum(lens[:i]) for i in range(len(lens))]

    def run():
        st, out = state.to(DEV), torch.empty(T, heads * vdim, dtype=dtype, device=DEV)
        ops.gated_recurrence(qfv.to(DEV), st, fb.to(DEV), low.to(DEV), nw.to(DEV), out, i32(list(range(len(lens)))), i32(starts), i32(lens),
                             len(lens), heads, d, vdim, 1e-5)
        return out.double().cpu(), st.double().cpu()

    out, st = run()
    monkeypatch.setattr(ops, "DECAY_CHUNKS_FROM", 1 << 30)
    walked, wst = run()
    x = qfv.double().to(DEV)
    q = x[:, :heads * d] * torch.sigmoid(x[:, :heads * d])
    f = low.double().to(DEV) + (1 - low.double().to(DEV)) * torch.sigmoid(x[:, heads * d:2 * heads * d] + fb.double().to(DEV))
    q, f, v = q.view(T, heads, d), f.view(T, heads, d), x[:, 2 * heads * d:].reshape(T, heads, vdim)
    for i, n in enumerate(lens):
        r = slice(starts[i], starts[i] + n)
        o, S = plain(q[r], 1 - f[r], v[r], f[r], torch.ones(n, heads, dtype=torch.float64, device=DEV),
                     torch.zeros(heads, dtype=torch.float64, device=DEV), state[i].double().to(DEV).transpose(1, 2))
        o = (o * torch.rsqrt(o.pow(2).mean(-1, keepdim=True) + 1e-5) * nw.double().to(DEV)).reshape(n, -1).cpu()
        S = S.transpose(1, 2).cpu()
        rel = lambda a, b: float((a - b).norm() / b.norm())  # noqa: E731
        bound = 16 * 2.0 ** -24 if dtype == torch.float32 else 2.0 ** -8
        assert rel(out[r], o) < bound and rel(st[i], S) < 16 * 2.0 ** -24
        assert rel(out[r], o) < 1.5 * rel(walked[r], o) + 2.0 ** -24 and rel(st[i], S) < 1.5 * rel(wst[i], S) + 2.0 ** -24
    assert torch.equal(st[-1].float(), state[-1])


NOT_FINITE = [("v", float("inf")), ("v", float("nan")), ("v", 3.4e38), ("k", float("-inf")), ("q", float("nan")), ("decay", float("nan")),
              ("state", float("inf"))]


@pytest.mark.parametrize("form,heads,groups,what,value", [
    (form, heads, groups, what, value) for form, heads, groups in (("head", 2, 1), ("token", 2, 2), ("channel", 2, 2))
    for what, value in NOT_FINITE if (form, what) != ("head", "decay")])  # (a constant a head has no token of its own)
@pytest.mark.parametrize("vdim", [64, 128])
def test_chunks_not_finite(form, heads, groups, vdim, what, value, monkeypatch):
    """One number that is not finite (or whose first bfloat16 is not): tokens ahead of it do not see it, those behind have what
    the walk gives them, and other requests and heads have the bits of a clean run."""
    from tokasaurus_b200.kernels import ops

    lens, hit, size = [200, 300, 260], 200 + 137, heads * vdim * 128  # the second request's third chunk, inside a block of 16
    p, state, ref = problem(form, heads, groups, vdim, lens, 11 + vdim)
    if form != "head":
        for name in ("dt_dec", "decay_vec"):  # (decays of zero would bury what is looked for)
            if p[name] is not None:
                p[name] = p[name].clamp(min=0.3)
    clean, cst = run(p, state, lens, heads, groups, vdim)
    head = heads - 1
    col = {"v": head * vdim + 5, "k": (groups - 1) * 128 + 3, "q": (groups - 1) * 128 + 3}
    bad, bstate = dict(p), state.clone()
    if what == "state":
        bstate[1, head * vdim * 128 + 77], hit = value, 200
    elif what == "decay":
        name = "dt_dec" if form == "token" else "decay_vec"
        bad[name] = p[name].clone()
        bad[name][hit, heads + head if form == "token" else head * 128 + 3] = value
    else:
        bad[what] = p[what].clone()
        bad[what][hit, col[what]] = value
    out, st = run(bad, bstate, lens, heads, groups, vdim)
    monkeypatch.setattr(ops, "DECAY_CHUNKS_FROM", 1 << 30)
    walked, wst = run(bad, bstate, lens, heads, groups, vdim)
    one = slice(head * vdim, (head + 1) * vdim)
    others = torch.ones(heads * vdim, dtype=torch.bool)
    others[one if groups > 1 or what in ("v", "state") else slice(None)] = False  # (heads that share q and k share their numbers)
    chunk0 = 200 + (hit - 200) // 64 * 64
    assert torch.equal(out[:chunk0], clean[:chunk0]) and torch.equal(out[500:], clean[500:])
    assert torch.equal(out[:, others], clean[:, others])
    near = lambda x, y: float((x.double() - y.double()).norm()) <= 16 * 2.0 ** -24 * float(y.double().norm())  # noqa: E731
    assert out[chunk0:hit].isfinite().all() and near(out[chunk0:hit], clean[chunk0:hit])
    assert (~walked[hit:500, one].isfinite()).any() or value == 3.4e38
    for got, want in ((out[hit:500], walked[hit:500]), (st[1], wst[1])):
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[got.isinf()], want[want.isinf()])
        assert torch.equal(got.isinf(), want.isinf())
        fine = want.isfinite()
        assert near(got[fine], want[fine])
    assert torch.equal(st[0], cst[0]) and torch.equal(st[2:], cst[2:])
    monkeypatch.undo()
    assert torch.equal(run(bad, bstate, lens, heads, groups, vdim, write=False)[0].nan_to_num(), out.nan_to_num())


@pytest.mark.parametrize("vdim", [64, 128])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3.4e38])
def test_chunks_of_the_forgetting_recurrence_not_finite(vdim, value, monkeypatch):
    """The same behind gates: a value that is not finite, in the middle of a block of 16 tokens."""
    from tokasaurus_b200.kernels import ops

    heads, d, lens, hit = 2, 128, [250, 1, 200], 101
    g = torch.Generator().manual_seed(vdim)
    T, starts = sum(lens), [0, 250, 251]
    qfv = torch.randn(T, heads * (2 * d + vdim), generator=g)
    fb, low = torch.randn(heads * d, generator=g), torch.rand(heads * d, generator=g) * 0.95
    nw = torch.rand(vdim, generator=g) + 0.5
    state = torch.randn(len(lens), heads, vdim, d, generator=g)

    def run(x):
        st, out = state.to(DEV), torch.empty(T, heads * vdim, device=DEV)
        ops.gated_recurrence(x.to(DEV), st, fb.to(DEV), low.to(DEV), nw.to(DEV), out, i32([0, 1, 2]), i32(starts), i32(lens), len(lens), heads, d,
                             vdim, 1e-5)
        return out.cpu(), st.cpu()

    clean, cst = run(qfv)
    x = qfv.clone()
    x[hit, 2 * heads * d + vdim + 9] = value  # the second head's
    out, st = run(x)
    monkeypatch.setattr(ops, "DECAY_CHUNKS_FROM", 1 << 30)
    walked, wst = run(x)
    near = lambda a, b: float((a.double() - b.double()).norm()) <= 64 * 2.0 ** -24 * float(b.double().norm())  # noqa: E731
    assert torch.equal(out[:64], clean[:64]) and torch.equal(out[250:], clean[250:]) and torch.equal(out[:, :vdim], clean[:, :vdim])
    assert out[64:hit].isfinite().all() and near(out[64:hit], clean[64:hit]) and torch.equal(st[1:], cst[1:])
    for got, want in ((out[hit:250], walked[hit:250]), (st[0], wst[0])):
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
        fine = want.isfinite()
        assert near(got[fine], want[fine])


@pytest.mark.parametrize("form,heads,groups", [("head", 2, 1), ("token", 2, 2), ("channel", 2, 2)])
@pytest.mark.parametrize("size", [1e-35, 1e-38, 1e27, 1e33])
def test_chunks_far_from_one(form, heads, groups, size, monkeypatch):
    """Values and states close to the smallest normal number, and so large that a cut number does not hold them: no less exact than the
    walk."""
    from tokasaurus_b200.kernels import ops

    lens = [260]
    p, state, _ = problem(form, heads, groups, 128, lens, 5)
    p["v"], state = p["v"] * size, state * size
    out, st = run(p, state, lens, heads, groups, 128)
    monkeypatch.setattr(ops, "DECAY_CHUNKS_FROM", 1 << 30)
    walked, wst = run(p, state, lens, heads, groups, 128)
    # the walk at another size by a power of two, where nothing under- or overflows
    up = 2.0 ** (100 if size < 1 else -100)
    p["v"], big = p["v"] * up, state * up
    ref, rst = run(p, big, lens, heads, groups, 128)
    monkeypatch.undo()
    n = heads * 128 * 128
    for got, walk, want in ((out, walked, ref), (st[0, :n], wst[0, :n], rst[0, :n])):
        want = want.double() / up
        err = lambda x: float((x.double() - want).norm() / want.norm())  # noqa: E731
        assert got.isfinite().all() and err(got) <= 1.5 * err(walk) + 16 * 2.0 ** -24


@pytest.mark.parametrize("lens,chunks", [([128] * 5, None), ([100, 191, 150], None), ([100, 200, 1, 321], 4 + 6)])
@pytest.mark.parametrize("layer", ["decayed", "forget"])
def test_a_step_s_layer_launches_what_its_requests_need(lens, chunks, layer, monkeypatch):
    """A layer of an eager step: no chunk kernel and no scratch without a long request, and scratch for the long ones alone."""
    from tokasaurus_b200.cache import CacheManager
    from tokasaurus_b200.engine.batch import Stager, StepContext, StepEntry, build_host_batch
    from tokasaurus_b200.engine.runtime import Runtime
    from tokasaurus_b200.kernels import ops
    from tokasaurus_b200 import parts as P

    H, W = 2, 256
    if layer == "decayed":
        part = P.DecayedLinearAttention(W, H, 128, 128, [0.9, 0.99], 1e-5, "q", "k", "v", "g", "norm", "o")
    else:
        part = P.GatedLinearRecurrence(W, H, 128, 128, 1e-5, "q", "k", "f_bias", "lower", "v", "norm", "o")
    g = torch.Generator().manual_seed(1)
    rt = Runtime.make(DEV, "bfloat16")
    part.bind({s.name: (torch.rand(s.shape, generator=g) * 0.5 if s.role == "vector" else torch.randn(s.shape, generator=g) / 16).to(
        DEV, torch.float32 if s.role == "vector" else torch.bfloat16) for s in part.weight_specs()}, rt)
    cm = CacheManager({0: part.cache_need()}, 16, 4, len(lens), dtype=rt.dtype, device=rt.device)
    for i, n in enumerate(lens):
        cm.admit(i)
        cm.ensure_capacity(i, n)
    ctx = StepContext(build_host_batch([StepEntry(i, [0] * n, 0, [n - 1]) for i, n in enumerate(lens)], cm), cm, rt.device, Stager(rt.device))
    h = torch.randn(sum(lens), W, generator=g).bfloat16().to(DEV)
    seen, real = [], ops._decay_chunks

    def spy(*args):
        out = real(*args)
        seen.append(out[1].shape[0])
        return out

    monkeypatch.setattr(ops, "_decay_chunks", spy)
    part.forward(ctx, h, cm.layer_cache(0))
    assert seen == ([] if chunks is None else [chunks])
    seen.clear()
    ctx.plan_caps = {}  # as while a step graph is recorded: what any step of the shape can need
    part.forward(ctx, h, cm.layer_cache(0))
    assert len(seen) == 1 and seen[0] >= (chunks or 0)
