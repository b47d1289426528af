"""The kernels of the 32-bit run alone: the float32 product and attention against float64, at the edges of their tiles,
and against themselves under other cuts of the same rows (a sum's order hangs on the operation's sizes only)."""

import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
EPS = 2.0 ** -24        # half a unit in the last place of float32


def _product(a, w, rows):
    from bare_cuda_4gib_b200.kernels import lib as K
    out = torch.full((rows, w.shape[0]), float("nan"), device=DEV)
    K.matmul_plain(a, w, out, rows)
    return out


@pytest.mark.parametrize("n,k", [(1, 4), (63, 36), (130, 300), (2560, 2048), (5000, 260), (300, 5632)])
def test_matmul_f32(n, k):
    torch.manual_seed(n + k)
    a, w = torch.randn(600, k, device=DEV), torch.randn(n, k, device=DEV)
    want, size = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    whole = _product(a, w, 600)
    # a segment's chains of packed FMAs, then the pair and the eight segments: each rounds once, relative to at most the sum of
    # the sizes
    segment = -(--(-k // 8) // 32) * 32
    assert ((whole.double() - want).abs() <= (segment / 2 + 1 + 8) * EPS * size).all()
    for rows in (1, 2, 3, 4, 5, 8, 9, 16, 17, 24, 25, 33, 64, 65, 100, 257):
        assert torch.equal(_product(a, w, rows), whole[:rows]), rows


def test_matmul_f32_strided_rows_and_bad_values():
    torch.manual_seed(3)
    wide = torch.randn(40, 2 * 64, device=DEV)
    a, w = wide[:, 64:], torch.randn(70, 64, device=DEV)
    wide[7, 70] = float("inf")
    wide[9, 65] = float("nan")
    got, clean = _product(a, w, 40), _product(a.contiguous(), w, 40)
    assert torch.equal(got.nan_to_num(7.0, 8.0, 9.0), clean.nan_to_num(7.0, 8.0, 9.0))
    bad = ~torch.isfinite(got).all(-1)
    assert bad.nonzero().flatten().tolist() == [7, 9]        # a row's values stay in that row


class _Attention:
    """Requests of (tokens of the step, keys) over pages in random order."""

    def __init__(self, dim, kv_heads, group, seqs, window, page):
        self.dim, self.kv_heads, self.group, self.window, self.page, self.seqs = dim, kv_heads, group, window, page, seqs
        blocks = -(-max(kv for _, kv in seqs) // page)
        self.elems = 2 * kv_heads * page * dim
        self.pool = torch.full((len(seqs) * blocks + 2, self.elems), float("nan"), device=DEV)    # pages nobody holds
        table = torch.full((len(seqs), blocks), -1, dtype=torch.int32)
        order = torch.randperm(self.pool.shape[0]).tolist()
        for s, (_, kv) in enumerate(seqs):
            for b in range(-(-kv // page)):
                table[s, b] = order.pop()
                self.pool[table[s, b]] = torch.randn(self.elems, device=DEV)
        self.table = table.to(DEV)
        self.q = torch.randn(sum(q for q, _ in seqs), kv_heads * group * dim, device=DEV)
        self.at = [sum(q for q, _ in seqs[:s]) for s in range(len(seqs))]

    def run(self, parts):
        """`parts`: (request, first token of its step, tokens); what the kernel gives for them as one step."""
        from bare_cuda_4gib_b200.kernels import attention_f32, lib as K
        ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
        ctx, lens = types.SimpleNamespace(), [n for _, _, n in parts]
        kv = [self.seqs[s][1] - self.seqs[s][0] + first + n for s, first, n in parts]
        ctx.host_q_len, ctx.n_seqs, ctx.max_q_len, ctx.n_tokens, ctx.stream = lens, len(parts), max(lens), sum(lens), K.stream_handle()
        ctx.seq_q_start, ctx.seq_q_len, ctx.seq_kv_len = ints([sum(lens[:i]) for i in range(len(lens))]), ints(lens), ints(kv)
        table = self.table[[s for s, _, _ in parts]].contiguous()
        view = K.CacheView(self.pool.data_ptr(), self.pool.data_ptr() + self.elems // 2 * 4, table, self.elems, table.stride(0),
                           self.page, self.kv_heads, self.dim, torch.float32)
        q = torch.cat([self.q[self.at[s] + first: self.at[s] + first + n] for s, first, n in parts])
        out = torch.full_like(q, float("nan"))
        assert attention_f32.takes(q, out, view)
        attention_f32.run(ctx, q, out, view, self.kv_heads * self.group, self.dim ** -0.5, self.window)
        return out

    def want(self, absent=()):
        """In 64 bits; `absent`: (request, page of it) whose keys count as not there."""
        rows = []
        for s, (n, kv) in enumerate(self.seqs):
            held = self.table[s, : -(-kv // self.page)].long()
            both = self.pool[held].view(-1, 2, self.kv_heads, self.page, self.dim).double()
            k, v = (both[:, i].permute(1, 0, 2, 3).reshape(self.kv_heads, -1, self.dim)[:, :kv] for i in (0, 1))
            q = self.q[self.at[s]: self.at[s] + n].double().view(n, self.kv_heads, self.group, self.dim)
            i, j = (kv - n + torch.arange(n, device=DEV))[:, None], torch.arange(kv, device=DEV)[None]
            hidden = (j > i) | (i - j >= self.window) if self.window else j > i
            for r, b in absent:
                hidden = hidden | (r == s) & (j // self.page == b)
            w = (torch.einsum("tkgd,kjd->kgtj", q, k) * self.dim ** -0.5).masked_fill(hidden, -float("inf")).softmax(-1)
            rows.append(torch.einsum("kgtj,kjd->tkgd", w, v).reshape(n, -1))
        return torch.cat(rows)


@pytest.mark.parametrize("dim,kv_heads,group,page,window,seqs", [
    (64, 2, 8, 64, 0, [(1, 300), (1, 1), (70, 70), (1, 64), (2, 65)]),
    (64, 2, 1, 32, 0, [(3, 70), (9, 64), (8, 8), (90, 200)]),            # at most and over eight rows of a request
    (64, 1, 3, 16, 40, [(3, 70), (1, 2100), (65, 129)]),                 # a window; more spans than a cluster holds at once
    (128, 2, 4, 64, 0, [(1, 1100), (2, 127), (33, 128)]),
    (128, 1, 16, 32, 100, [(1, 333), (50, 90)]),                         # more than eight heads to a key head
])
def test_attention_f32(dim, kv_heads, group, page, window, seqs):
    torch.manual_seed(dim + group)
    case = _Attention(dim, kv_heads, group, seqs, window, page)
    whole, want = case.run([(s, 0, n) for s, (n, _) in enumerate(seqs)]), case.want()
    # scores of size ~ 4 carry dim / 2 + 2 roundings, which the exponential passes on; 64 values and a join a span follow
    bound = (4 * (dim / 2 + 2) + 2 * 64 + 3 * (max(kv for _, kv in seqs) / 64 + 1)) * EPS
    assert ((whole.double() - want).abs() <= bound * want.abs().max()).all()
    for tail in (1, 2, 7):                   # the last tokens of every request alone, as later steps would bring them
        parts = [(s, max(0, n - tail), min(n, tail)) for s, (n, _) in enumerate(seqs)]
        rows = torch.cat([whole[case.at[s] + f: case.at[s] + f + n] for s, f, n in parts])
        assert torch.equal(case.run(parts), rows), tail


@pytest.mark.parametrize("dim,kv", [(64, 4200), (128, 3100)])
def test_attention_f32_of_more_spans_than_the_cluster_holds_twice(dim, kv):
    """A few rows over three rounds of the cluster's spans, whose states are written again each time: against 64 bits, and the
    same bits every time and for the row alone."""
    torch.manual_seed(dim)
    case = _Attention(dim, 4, 2, [(1, kv), (3, kv - 70), (1, 2), (4, kv - 1)], 0, 64)
    parts = [(s, 0, n) for s, (n, _) in enumerate(case.seqs)]
    got, want = case.run(parts), case.want()
    bound = (4 * (dim / 2 + 2) + 2 * 64 + 3 * (kv / 64 + 1)) * EPS          # as in test_attention_f32
    assert ((got.double() - want).abs() <= bound * want.abs().max()).all()
    for _ in range(20):
        assert torch.equal(case.run(parts), got)
    assert torch.equal(case.run([(3, 3, 1)]), got[-1:])


@pytest.mark.parametrize("rows,hidden,partials", [(1, 64, 1), (3, 2048, 2), (300, 4100, 1), (2, 2050, 1)])
def test_add_rmsnorm_f32(rows, hidden, partials):
    from bare_cuda_4gib_b200.kernels import lib as K
    torch.manual_seed(hidden)
    x, w = torch.randn(rows, hidden, device=DEV), 1.0 + 0.1 * torch.randn(hidden, device=DEV)
    delta = torch.randn(partials, rows, hidden, device=DEV)
    residual, out = x.clone(), torch.empty(rows, hidden, device=DEV)
    K.add_rmsnorm(residual, K.Partials(delta if partials > 1 else delta[0], partials), w, out, 1e-5, rows)
    want = x.double() + delta.double().sum(0)
    normed = want / torch.sqrt((want * want).mean(-1, keepdim=True) + 1e-5) * w.double()
    assert ((residual.double() - want).abs() <= (partials + 1) * 2 * EPS * (x.abs() + delta.abs().sum(0)).double()).all()
    # the sum of squares adds up at most 16 terms a thread and 10 levels of the block, the factor rounds four times more
    assert ((out.double() - normed).abs() <= ((16 + 10) / 2 + 6 + 2 * partials) * 2 * EPS * normed.abs() + 1e-6).all()


def test_attention_f32_keeps_nan_in_its_row():
    """A query of NaN gives a row of NaN, whether its keys fill a span or not, and no other row changes."""
    torch.manual_seed(9)
    seqs = [(1, 10), (1, 300), (2, 128), (70, 70), (66, 200)]
    case = _Attention(64, 1, 4, seqs, 0, 32)
    parts = [(s, 0, n) for s, (n, _) in enumerate(seqs)]
    clean = case.run(parts)
    bad = [0, 1, 3, case.at[3], case.at[3] + 64, case.at[4] + 5]
    case.q[bad] = float("nan")
    got = case.run(parts)
    assert got[bad].isnan().all()
    others = [r for r in range(clean.shape[0]) if r not in bad]
    assert torch.equal(got[others], clean[others])


def test_attention_f32_of_infinite_values_hangs_on_the_row_alone():
    """Values of infinity behind keys whose weights underflow to zero: a row comes out finite or not by what it sees, not by
    the rows beside it in a step, and finite here, as the plain kernel has it."""
    from bare_cuda_4gib_b200.kernels import lib as K
    torch.manual_seed(10)
    seqs = [(1, 200), (70, 200), (130, 130)]
    case = _Attention(64, 1, 2, seqs, 0, 32)
    case.q.view(-1, 2, 64)[:, :, 0] = 8.0          # scores (8 k[0] / 8 and about 1 from the rest): 150 at key 5, -100 and -130 at two
    for s, (_, kv) in enumerate(seqs):
        for key in range(kv):
            page = case.pool[case.table[s, key // 32].long()].view(2, 32, 64)
            page[0, key % 32, 0] = {5: 150.0, 7: -100.0, 75: -130.0}.get(key, 0.0)
            if key in (7, 75, 80):                 # beside key 5; beside the keys of its own span; a span that key 5 puts out
                page[1, key % 32] = float("inf")
    parts = [(s, 0, n) for s, (n, _) in enumerate(seqs)]
    whole = case.run(parts)
    for first, n in ((129, 1), (100, 3), (70, 40)):
        assert torch.equal(case.run([(2, first, n)]), whole[case.at[2] + first: case.at[2] + first + n])
    plain = torch.empty_like(case.q)
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    view = K.CacheView(case.pool.data_ptr(), case.pool.data_ptr() + case.elems // 2 * 4, case.table, case.elems, case.table.stride(0), 32, 1, 64, torch.float32)
    K.attention_plain(case.q, plain, view, ints([kv - n + i for n, kv in seqs for i in range(n)]), ints([s for s, (n, _) in enumerate(seqs) for _ in range(n)]),
                      2, case.q.shape[0], 64 ** -0.5, 0)
    assert torch.isfinite(plain).all() and torch.isfinite(whole).all()


@pytest.mark.parametrize("dim,kv_heads,group,page,window", [(64, 2, 2, 16, 40), (64, 1, 8, 64, 100), (128, 1, 4, 32, 0), (64, 2, 1, 32, 300)])
def test_attention_f32_of_pages_that_are_not_held(dim, kv_heads, group, page, window):
    """Pages behind the window of all of a request's rows are given back (no entry in the table, and NaN where they were), and a
    page inside the window that is not held counts as absent: in the walk and in the cluster's form, at every cut."""
    torch.manual_seed(dim + page)
    seqs = [(1, 500), (2, 300), (70, 400), (33, 333)]            # (one or two tokens: the cluster's form; over eight rows: the walk)
    case = _Attention(dim, kv_heads, group, seqs, window, page)
    absent = [(s, (kv - 5) // page - 1) for s, (_, kv) in enumerate(seqs)]       # seen by the last rows, not held
    want = case.want(absent)
    gone = absent + [(s, b) for s, (n, kv) in enumerate(seqs) if window for b in range(max(0, kv - n - window + 1) // page)]
    assert len(gone) > len(absent) + 5 or not window
    for s, b in gone:
        case.pool[case.table[s, b].long()] = float("nan")
        case.table[s, b] = -1
    whole = case.run([(s, 0, n) for s, (n, _) in enumerate(seqs)])
    bound = (4 * (dim / 2 + 2) + 2 * 64 + 3 * (500 / 64 + 1)) * EPS          # as in test_attention_f32
    assert ((whole.double() - want).abs() <= bound * want.abs().max()).all()
    for tail in (1, 30):
        parts = [(s, max(0, n - tail), min(n, tail)) for s, (n, _) in enumerate(seqs)]
        assert torch.equal(case.run(parts), torch.cat([whole[case.at[s] + f: case.at[s] + f + n] for s, f, n in parts])), tail


def test_attention_f32_of_more_requests_than_a_grid_has_layers():
    from bare_cuda_4gib_b200.kernels import attention_f32, lib as K
    torch.manual_seed(12)
    n, page, held = 65535 + 9, 16, 40
    pool, q = torch.randn(held, 2, page, 64, device=DEV), torch.randn(n, 64, device=DEV)
    ints = lambda x: x.to(device=DEV, dtype=torch.int32)
    pages, kv = torch.randint(held, (n,)), torch.randint(1, page + 1, (n,))
    table, ctx = ints(pages)[:, None].contiguous(), types.SimpleNamespace()
    ctx.host_q_len, ctx.n_seqs, ctx.max_q_len, ctx.n_tokens, ctx.stream = [1] * n, n, 1, n, K.stream_handle()
    ctx.seq_q_start, ctx.seq_q_len, ctx.seq_kv_len = ints(torch.arange(n)), ints(torch.ones(n)), ints(kv)
    view = K.CacheView(pool.data_ptr(), pool[0, 1].data_ptr(), table, 2 * page * 64, 1, page, 1, 64, torch.float32)
    out = torch.full_like(q, float("nan"))
    attention_f32.run(ctx, q, out, view, 1, 0.125, 0)
    keys = pool[pages.to(DEV)].double()
    hidden = torch.arange(page, device=DEV)[None] >= kv.to(DEV)[:, None]
    w = (torch.einsum("nd,njd->nj", q.double(), keys[:, 0]) * 0.125).masked_fill(hidden, -float("inf")).softmax(-1)
    want = torch.einsum("nj,njd->nd", w, keys[:, 1])
    assert ((out.double() - want).abs() <= (4 * 34 + 2 * 64 + 6) * EPS * want.abs().max()).all()
