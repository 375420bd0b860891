"""Prompt portions over cached rows on the tcgen05 kernel against float64 sums: latent rows and [k | v] rows, groups of heads that
do and do not divide a block's 128 rows, portions behind cached tokens, windows and chunks that start inside a tile, pages that
come as TMA boxes and pages that are gathered, scores far beyond the cap, factors below zero, sinks, gates and sigmoid weights."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


class Problem:
    """Requests with cached rows (the step's own among them) on shuffled pages; what no request owns is no number."""

    def __init__(self, row, nkv, ps, lens, new, seed):
        g = torch.Generator().manual_seed(seed)
        pages = [-(-n // ps) for n in lens]
        n_pages = sum(pages) + 3
        perm = torch.randperm(n_pages, generator=g).tolist()
        cache = torch.full((n_pages, nkv, ps, row), math.nan)
        self.rows, table, indptr = [], [], [0]
        for n, np_ in zip(lens, pages):
            mine = [perm.pop() for _ in range(np_)]
            rows = torch.randn(n, nkv, row, generator=g).bfloat16().float()
            for j in range(n):
                cache[mine[j // ps], :, j % ps] = rows[j]
            table += mine
            indptr.append(len(table))
            self.rows.append(rows.to(DEV))
        self.cache, self.lens, self.new, self.nkv, self.ps = cache.bfloat16().to(DEV), lens, new, nkv, ps
        self.start = [sum(new[:i]) for i in range(len(new))]
        self.T = sum(new)
        self.tables = dict(seq_q_start=i32(self.start), seq_q_len=i32(new), seq_kv_len=i32(lens), page_indptr=i32(indptr), page_ids=i32(table))
        self.g = g

    def want(self, q, kd, v0, vd, heads, scale, window=0, chunk=0, cap=0.0, sinks=None, head_scale=None, head_bias=None, sigmoid=False):
        out = torch.zeros(self.T, heads, vd, dtype=torch.float64, device=DEV)
        group = heads // self.nkv
        for s, (n, L) in enumerate(zip(self.new, self.lens)):
            r = self.rows[s].double()
            k, v = (x.repeat_interleave(group, 1) for x in (r[..., :kd], r[..., v0:v0 + vd]))
            qq = q[self.start[s]:self.start[s] + n].double().view(n, heads, kd)
            y = torch.einsum("thd,shd->hts", qq, k) * scale
            if head_scale is not None:
                y = y * head_scale.double()[:, None, None]
            if cap:
                y = cap * torch.tanh(y / cap)
            if head_bias is not None:
                y = y + head_bias.double()[:, None, None]
            i = torch.arange(L - n, L, device=DEV)[:, None]
            j = torch.arange(L, device=DEV)[None, :]
            see = j <= i
            if window:
                see &= j > i - window
            if chunk:
                see &= j >= i - i % chunk
            if sigmoid:
                w = torch.sigmoid(y) * see
            else:
                y = y.masked_fill(~see, -math.inf)
                top = y.amax(-1, keepdim=True)
                if sinks is not None:
                    top = torch.maximum(top, sinks.double()[:, None, None])
                w = torch.exp(y - top)
                den = w.sum(-1, keepdim=True) + (torch.exp(sinks.double()[:, None, None] - top) if sinks is not None else 0)
                w = w / den
            out[self.start[s]:self.start[s] + n] = torch.einsum("hts,shv->thv", w, v)
        return out


def check(got, want, several, magnitude):
    """Weights are rounded to bfloat16 for their product with the values and the result once more: 2^-9 of the sum of
    |weight value|, which is at most ``magnitude``, and 2^-9 of the result, doubled for what the score loses."""
    err = (got.double() - want)[several].abs()
    assert err.max() <= 2.0 ** -7 * magnitude, (float(err.max()), magnitude)
    assert err.norm() <= 6e-3 * want[several].norm()


@pytest.mark.parametrize("row,vd,heads", [(256, 192, 16), (256, 192, 32), (256, 128, 5), (128, 64, 128), (192, 96, 1)])
@pytest.mark.parametrize("window,ps", [(0, 16), (100, 16), (64, 128), (300, 12)])
def test_latent_rows(row, vd, heads, window, ps):
    from tokasaurus_b200.kernels import ops

    (module,) = ops.rows_tc_modules(row, row, 0, vd, False)
    p = Problem(row, 1, ps, [37, 200, 1, 449], [37, 71, 1, 130], heads + window)
    q = torch.randn(p.T, heads * row, generator=p.g).bfloat16().to(DEV)
    out = torch.full((p.T, heads * row), 7.0, dtype=torch.bfloat16, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    scale = 1 / math.sqrt(row)
    ops.attn_rows_tc(module, q, out, row, p.cache, **p.tables, n_seqs=4, n_heads=heads, n_kv_heads=1, page_size=ps, scale=scale,
                     window=window, status=status)
    want = p.want(q, row, 0, vd, heads, scale, window)
    several = torch.ones(p.T, dtype=torch.bool, device=DEV)
    several[p.start[2]] = False
    got = out.view(p.T, heads, row)
    assert int(status) == 0
    check(got[..., :vd], want, several, 4.5)
    assert (got[..., vd:] == 7).all() and (got[~several] == 7).all()  # nothing beside the values, nothing of a single token


@pytest.mark.parametrize("dim,vdim,heads,nkv", [(64, 64, 8, 2), (128, 128, 4, 4), (128, 64, 6, 2)])
@pytest.mark.parametrize("window,chunk,ps", [(0, 0, 16), (100, 0, 16), (65, 0, 4), (0, 96, 16)])
@pytest.mark.parametrize("form", ["plain", "capped", "far", "heads", "sigmoid"])
def test_key_value_rows(dim, vdim, heads, nkv, window, chunk, ps, form):
    from tokasaurus_b200.kernels import ops

    p = Problem(dim + vdim, nkv, ps, [300, 64, 1, 129], [172, 64, 1, 2], dim + vdim + window + len(form))
    q = torch.randn(p.T, heads * dim, generator=p.g).bfloat16().to(DEV)
    scale = dim ** -0.5
    opt = {}
    vec = lambda f: f(torch.randn(heads, generator=p.g)).to(DEV)  # noqa: E731
    if form == "capped":  # scores well within the cap: the polynomial; with sinks and an output gate
        opt = dict(softcap=50.0, sinks=vec(lambda x: 3 * x))
    if form == "far":  # scores many times the cap
        opt, scale = dict(softcap=4.0, sinks=vec(lambda x: x)), scale * 8
    if form == "heads":
        opt = dict(head_scale=vec(lambda x: x), head_bias=vec(lambda x: x), softcap=6.0)
    if form == "sigmoid":
        opt = dict(head_bias=vec(lambda x: x), sigmoid=True)
    gate = torch.randn(p.T, heads, generator=p.g).to(DEV) if form == "capped" else None
    out = torch.full((p.T, heads * vdim), 7.0, dtype=torch.bfloat16, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    (module,) = ops.sink_rows_tc_modules(dim, vdim)
    ops.attn_rows_tc(module, q, out, vdim, p.cache, **p.tables, n_seqs=4, n_heads=heads, n_kv_heads=nkv, page_size=ps, scale=scale,
                     window=window, status=status, chunk=chunk, gate=gate, out_scale=0.5, **opt)
    names = dict(softcap="cap")
    want = 0.5 * p.want(q, dim, dim, vdim, heads, scale, window, chunk, **{names.get(k, k): v for k, v in opt.items()})
    if gate is not None:
        want = want * torch.sigmoid(gate.double())[..., None]
    several = torch.ones(p.T, dtype=torch.bool, device=DEV)
    several[p.start[2]] = False
    assert int(status) == 0
    keys = min(300, window or 300, chunk or 300)
    check(out.view(p.T, heads, vdim), want, several, 2.5 * (0.5 * keys ** 0.5 if form == "sigmoid" else 1.0) * (2 if form == "sigmoid" else 1))
    assert (out.view(p.T, heads, vdim)[~several] == 7).all()


def test_what_it_refuses():
    """A sink beside sigmoid weights would scale the result, and vectors of other sizes would be read out of range."""
    from tokasaurus_b200.kernels import ops

    p = Problem(128, 2, 16, [90, 64], [30, 64], 5)
    q = torch.randn(p.T, 8 * 64, generator=p.g).bfloat16().to(DEV)
    out, status = torch.empty_like(q), torch.zeros(1, dtype=torch.int32, device=DEV)
    (module,) = ops.sink_rows_tc_modules(64, 64)
    vec = lambda n, t=torch.float32: torch.zeros(n, dtype=t, device=DEV)  # noqa: E731
    for opt in (dict(sigmoid=True, sinks=vec(8)), dict(sinks=vec(7)), dict(head_scale=vec(8, torch.float64)), dict(head_bias=vec(4)),
                dict(gate=torch.zeros(p.T - 1, 8, device=DEV))):
        with pytest.raises(ops.KernelError):
            ops.attn_rows_tc(module, q, out, 64, p.cache, **p.tables, n_seqs=2, n_heads=8, n_kv_heads=2, page_size=16, scale=0.1,
                             window=None, status=status, **opt)


def test_the_step_takes_it():
    """``attn_sink_tc``: portions on this kernel, single tokens on theirs; forms that it does not have stay where they were."""
    from tokasaurus_b200.kernels import ops

    p = Problem(128, 2, 16, [300, 64, 90], [172, 64, 1], 5)
    q = torch.randn(p.T, 8 * 64, generator=p.g).bfloat16().to(DEV)
    sinks = torch.randn(8, generator=p.g).to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = torch.empty(p.T, 8 * 64, dtype=torch.bfloat16, device=DEV)
    ops.attn_sink_tc(q, out, p.cache, **p.tables, n_seqs=3, sinks=sinks, n_heads=8, n_kv_heads=2, dim=64, vdim=64, page_size=16,
                     scale=0.125, softcap=30.0, window=100, status=status)
    want = p.want(q, 64, 64, 64, 8, 0.125, 100, 0, 30.0, sinks)
    check(out.view(p.T, 8, 64), want, torch.ones(p.T, dtype=torch.bool, device=DEV), 2.5)
    assert ops.sink_rows_tc_modules(64, 64, maps=2) == ops.sink_rows_tc_modules(64, 64, distance=True) == ()
    assert ops.sink_rows_tc_modules(64, 64, keep_first=4) == ops.sink_rows_tc_modules(48, 64) == ops.sink_rows_tc_modules(64, 256) == ()


@pytest.mark.parametrize("dim", [64, 48])  # on this kernel, on the mma.sync one
def test_a_gate_with_more_rows_than_tokens(dim):
    """The gate's logits as a column slice of a taller and wider tensor: ``attn_sink_tc`` takes the first rows."""
    from tokasaurus_b200.kernels import ops

    p = Problem(2 * dim, 2, 16, [300, 64, 90], [172, 64, 1], 5)
    q = torch.randn(p.T, 8 * dim, generator=p.g).bfloat16().to(DEV)
    wide = torch.randn(p.T + 19, 20, generator=p.g).to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)

    def run(gate):
        out = torch.empty(p.T, 8 * dim, dtype=torch.bfloat16, device=DEV)
        ops.attn_sink_tc(q, out, p.cache, **p.tables, n_seqs=3, sinks=None, n_heads=8, n_kv_heads=2, dim=dim, vdim=dim, page_size=16,
                         scale=0.125, softcap=None, window=100, status=status, gate=gate)
        return out

    assert torch.equal(run(wide[:, 7:15]), run(wide[:p.T, 7:15].contiguous()))
    for bad in (wide[:p.T - 1, 7:15], wide[:, 7:14], wide[:, 7:15].double(), wide.T[7:15, :p.T].T[:, :8].T.contiguous().T):
        with pytest.raises(ops.KernelError):
            run(bad)


def test_more_tiles_than_a_grid_has_rows():
    """128 heads a kv head are a block a token: a step of more tokens than 65,535, which the mma.sync kernel took."""
    from tokasaurus_b200.kernels import ops

    T, heads, row, ps, window = 66000, 128, 128, 16, 40
    (module,) = ops.rows_tc_modules(row, row, 0, 64, False)
    g = torch.Generator(DEV).manual_seed(1)
    pages = -(-T // ps)
    cache = torch.randn(pages, 1, ps, row, generator=g, device=DEV).bfloat16()
    q = torch.randn(T, heads * row, generator=g, device=DEV, dtype=torch.bfloat16)
    out = torch.full((T, heads * 64), 7.0, dtype=torch.bfloat16, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.attn_rows_tc(module, q, out, 64, cache, i32([0]), i32([T]), i32([T]), i32([0, pages]), i32(range(pages)), n_seqs=1,
                     n_heads=heads, n_kv_heads=1, page_size=ps, scale=0.1, window=window, status=status)
    assert int(status) == 0
    flat = cache.view(-1, row)
    for t in (0, 17, 40000, 65535, 65536, T - 1):
        rows = flat[max(0, t - window + 1):t + 1].double()
        w = torch.softmax(q[t].view(heads, row).double() @ rows.T * 0.1, -1)
        check(out[t].view(1, heads, 64), (w @ rows[:, :64])[None], torch.ones(1, dtype=torch.bool, device=DEV), 4.5)


@pytest.mark.parametrize("ps", [16, 12])  # pages that come as TMA boxes, pages that are gathered
@pytest.mark.parametrize("form", ["latent", "key_value"])
def test_pages_given_back_and_pages_beyond_the_pool(ps, form):
    """Pages behind the window (id -1) are not looked at; an id beyond the pool sets the status bit, its keys' values count for nothing,
    and no other request sees anything of it."""
    from tokasaurus_b200.kernels import ops

    kd, v0, vd, nkv, heads, window = (256, 0, 192, 1, 16, 100) if form == "latent" else (64, 64, 64, 3, 12, 100)
    row = 256 if form == "latent" else 128
    (module,) = ops.rows_tc_modules(row, kd, v0, vd, form != "latent")
    p = Problem(row, nkv, ps, [400, 333, 90], [70, 129, 90], ps)
    q = torch.randn(p.T, heads * kd, generator=p.g).bfloat16().to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)

    def run(ids):
        out = torch.full((p.T, heads * vd), 7.0, dtype=torch.bfloat16, device=DEV)
        ops.attn_rows_tc(module, q, out, vd, p.cache, **{**p.tables, "page_ids": ids}, n_seqs=3, n_heads=heads, n_kv_heads=nkv,
                         page_size=ps, scale=kd ** -0.5, window=window, status=status)
        return out

    whole = run(p.tables["page_ids"])
    check(whole.view(p.T, heads, vd), p.want(q, kd, v0, vd, heads, kd ** -0.5, window), torch.ones(p.T, dtype=torch.bool, device=DEV), 4.5)
    ids = p.tables["page_ids"].clone()
    first = (400 - 70 - window + 1) // ps  # the first page that request 0's portion sees
    ids[:first] = -1
    assert torch.equal(run(ids), whole) and int(status) == 0
    at = int(p.tables["page_indptr"][1]) + 250 // ps
    ids[at] = p.cache.shape[0] + 5
    out = run(ids)
    assert int(status) == 2  # a page id outside the pool
    mine = slice(p.start[1], p.start[1] + 129)
    assert torch.equal(out[: p.start[1]], whole[: p.start[1]]) and torch.equal(out[p.start[2]:], whole[p.start[2]:])
    assert out[mine].isfinite().all() and not torch.equal(out[mine], whole[mine])
