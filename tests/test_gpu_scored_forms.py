"""Attention with shaped scores in bfloat16 on the tensor cores, prompt rows and single-token rows, against the formula in 64 bits and against
the CUDA-core kernel: sequences that end one row before and after a tile and a page, pages in any order with no number in the places that no
row has reached, every shaping of a score, one to many heads of a group, values of 8 to 256 entries."""
import pytest
import torch

from kvad_b200.ops import Ops, lib

pytestmark = pytest.mark.gpu
PAGE = 64


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


class Case:
    """A paged cache, queries for the last `new` of each sequence's positions, and the exact answer with a bound on the error."""

    def __init__(self, seqs, H, G, dk, dv, *, alias=False, key_maps=1, cap=0.0, span=0.0, window=0, keep=0, chunk=0, gate=None, sinks=False, seed=0):
        g = torch.Generator(device="cuda")
        g.manual_seed(seed + dk * 7 + dv)
        rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
        self.seqs, self.H, self.dv, self.alias, self.scale = seqs, H, dv, alias, 1.5 / dk ** 0.5
        width = -(-max(c + n for c, n in seqs) // PAGE)
        n_pages = width * len(seqs) + 2
        order = torch.randperm(n_pages, generator=torch.Generator().manual_seed(seed + 3))
        self.table = order[:width * len(seqs)].reshape(len(seqs), width).to(torch.int32).cuda().contiguous()
        self.kp = torch.full((n_pages, G, PAGE, dk), float("nan"), dtype=torch.bfloat16, device="cuda")
        self.vp = None if alias else torch.full((n_pages, G // key_maps, PAGE, dv), float("nan"), dtype=torch.bfloat16, device="cuda")
        n_rows = sum(n for _, n in seqs)
        self.q = rnd(n_rows, H * dk + 8)[:, :H * dk]
        self.gate = {None: None, "entry": rnd(n_rows, H * dv), "head": rnd(n_rows, H)}[gate]
        self.sinks = torch.randn(H, generator=g, device="cuda") if sinks else None
        self.kw = dict(softcap=cap, slope_span=span, window=window, keep_first=keep, chunk=chunk, key_maps=key_maps, sinks=self.sinks, gate=self.gate,
                       value_dim=dv if alias else None)
        want, slack, at = [], [], 0
        for s, (cached, new) in enumerate(seqs):
            L = cached + new
            k = rnd(G, L, dk)
            v = k[:, :, :dv] if alias else rnd(G // key_maps, L, dv)
            for p in range(-(-L // PAGE)):
                n = min(PAGE, L - p * PAGE)
                self.kp[self.table[s, p].long(), :, :n] = k[:, p * PAGE:p * PAGE + n]
                if not alias:
                    self.vp[self.table[s, p].long(), :, :n] = v[:, p * PAGE:p * PAGE + n]
            kd = k.double().repeat_interleave(H // G, 0)
            vd = v.double().repeat_interleave(key_maps, 0).repeat_interleave(H // G, 0)
            qd = self.q[at:at + new].double().reshape(new, H, dk).transpose(0, 1)
            x = qd @ kd.transpose(1, 2) * self.scale
            # a score's error: the tensor core truncates after every 16 products (2^-22 of the sum of magnitudes a step is generous); the cap rounds what it
            # gives, which is no larger than the score and the cap, a few times
            ds = (qd.abs() @ kd.abs().transpose(1, 2)).max().item() * self.scale * (dk / 16 + 2) * 2.0 ** -22
            if cap:
                ds += min(cap, x.abs().max().item()) * 2.0 ** -21
                x = cap * torch.tanh(x / cap)
            pos, key = torch.arange(cached, L, device="cuda"), torch.arange(L, device="cuda")
            if span:
                slopes = 2.0 ** (-span * torch.arange(1, H + 1, device="cuda", dtype=torch.float64) / H)
                x = x - slopes[:, None, None] * (pos[:, None] - key[None, :])
                ds += span and L * 2.0 ** -22
            seen = key[None, :] <= pos[:, None]
            if window:
                seen &= (key[None, :] > pos[:, None] - window) | (key[None, :] < keep)
            if chunk:
                seen &= key[None, :] >= (pos - pos % chunk)[:, None]
            x = x.masked_fill(~seen, float("-inf"))
            if sinks:
                x = torch.cat([x, self.sinks.double()[:, None, None].expand(H, new, 1)], 2)
            p = torch.softmax(x, 2)[:, :, :L]
            f = 1.0 if gate is None else torch.sigmoid(self.gate[at:at + new].double().reshape(new, H, -1)).transpose(0, 1)
            want.append(((p @ vd) * f).transpose(0, 1).reshape(new, H * dv))
            # a weight's relative error: twice the scores', 2^-16 for its pieces, and 2^-17 for sums of up to L terms and exponentials of up to 2^7
            slack.append(((p @ vd.abs()) * f * (2 * ds + 2.0 ** -15)).transpose(0, 1).reshape(new, H * dv))
            at += new
        self.want, self.slack = torch.cat(want), torch.cat(slack)
        starts = [0]
        for _, n in seqs:
            starts.append(starts[-1] + n)
        self.starts, self.lens, self.max_new = i32(starts), i32([c + n for c, n in seqs]), max(n for _, n in seqs)

    def run(self, ops, out_dtype=torch.bfloat16, **extra):
        out = torch.full((self.q.shape[0], self.want.shape[1] + 8), float("nan"), dtype=out_dtype, device="cuda")
        ops.attention_scored(self.q, out[:, :-8], self.starts, self.lens, len(self.seqs), self.max_new, self.table, self.kp, self.vp, self.H, self.scale,
                             **self.kw, **extra)
        torch.cuda.synchronize()
        assert out[:, -8:].isnan().all()                  # nothing is written beside the heads
        return out[:, :-8].double()

    def check(self, got, out_dtype=torch.bfloat16):
        bound = self.slack + (2.0 ** -8 if out_dtype == torch.bfloat16 else 2.0 ** -23) * self.want.abs() + 1e-30
        worst = ((got - self.want).abs() / bound).max().item()
        assert worst <= 1.0, worst


EDGES = [(0, 129), (63, 2), (200, 65), (5, 1), (0, 64), (1, 127)]
SHAPES = [
    (4, 4, 64, 64, {}),                                                       # one head a group: a tile of 128 tokens
    (16, 1, 96, 96, dict(alias=True)),
    (16, 1, 256, 256, dict(alias=True, gate="entry")),                        # a latent of 256
    (4, 2, 256, 256, {}),                                                     # no room for two halves
    (2, 1, 400, 64, dict(alias=True)),
    (6, 2, 72, 40, dict(cap=30.0)),                                           # three heads a group, sizes that fill no 16
    (8, 2, 128, 128, dict(window=50, keep=4, gate="entry")),
    (20, 1, 64, 8, dict(window=1)),                                           # every row sees itself alone
    (12, 4, 32, 192, dict(chunk=96, sinks=True)),
    (4, 2, 128, 64, dict(span=8.0, gate="head")),
    (8, 8, 64, 64, dict(key_maps=2)),
    (2, 1, 8, 8, dict(sinks=True, window=130, keep=70, cap=5.0, span=4.0)),
]


@pytest.mark.parametrize("H,G,dk,dv,form", SHAPES)
def test_prompt_rows_on_the_tensor_cores(H, G, dk, dv, form):
    ops, cores = Ops(torch.bfloat16), Ops(torch.bfloat16)
    cores.scored_prompt = False
    c = Case(EDGES, H, G, dk, dv, **form)
    outs = [torch.bfloat16] if c.gate is not None or dv > 128 else [torch.bfloat16, torch.float32]
    for out in outs:
        assert lib("attention_scored_prompt").kvad_attention_scored_prompt_takes(dk, dv, int(c.alias), int(out == torch.float32)) == 1
        for o in (ops, cores):
            c.check(c.run(o, out), out)


@pytest.mark.parametrize("dk,dv,shift", [(64, 264, 0), (20, 16, 0), (64, 64, 4)])
def test_prompt_rows_it_does_not_take_go_to_the_cuda_cores(dk, dv, shift):
    """Values, keys and addresses out of its range: the same answer as with the tensor cores off, to the last bit."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").to(torch.bfloat16)
    q, kp, vp = rnd(70, 2 * dk + 8)[:, shift:shift + 2 * dk], rnd(3, 1, PAGE, dk), rnd(3, 1, PAGE, dv)
    outs = []
    for on in (True, False):
        ops = Ops(torch.bfloat16)
        ops.scored_prompt = on
        out = torch.full((70, 2 * dv), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.attention_scored(q, out, i32([0, 70]), i32([80]), 1, 70, i32([[2, 0, 1]]), kp, vp, 2, 0.1)
        outs.append(out)
    assert torch.equal(*outs) and outs[0].isfinite().all()


STEPS = [(0, 1), (63, 1), (64, 1), (129, 1), (700, 1), (191, 1)]


@pytest.mark.parametrize("splits", [1, 3, 16])
@pytest.mark.parametrize("H,G,dk,dv,form", SHAPES + [(16, 4, 64, 64, dict(cap=30.0, window=512, keep=4)), (17, 1, 40, 136, {}), (40, 1, 64, 64, dict(span=8.0))])
def test_single_token_rows_on_the_tensor_cores(H, G, dk, dv, form, splits):
    ops = Ops(torch.bfloat16)
    c = Case(STEPS, H, G, dk, dv, **form)
    scratch = torch.full((len(STEPS) * H * splits * (dv + 2),), float("nan"), device="cuda")
    for out in (torch.bfloat16, torch.float32):
        if out == torch.float32 and c.gate is not None:
            continue
        for per_block in (1, min(H // G, 32)):
            c.check(c.run(ops, out, n_splits=splits, scratch=scratch, heads_per_block=per_block), out)


def paged(k, v, order_seed=1):
    """One sequence's keys [G, L, dk] and values (None: the keys' first entries) as pages in any order, with its page table."""
    G, L, _ = k.shape
    n = -(-L // PAGE)
    order = torch.randperm(n, generator=torch.Generator().manual_seed(order_seed))
    table = order.to(torch.int32).cuda()[None].contiguous()

    def pages(x):
        out = torch.full((n, G, PAGE, x.shape[2]), float("nan"), dtype=torch.bfloat16, device="cuda")
        for p in range(n):
            m = min(PAGE, L - p * PAGE)
            out[order[p], :, :m] = x[:, p * PAGE:p * PAGE + m]
        return out
    return pages(k), None if v is None else pages(v), table


@pytest.mark.parametrize("H,dk,dv,alias", [(1, 64, 64, False), (16, 32, 32, False), (4, 128, 128, False), (2, 224, 192, True), (16, 288, 256, True)])
def test_prompt_weights_keep_their_32_bits(H, dk, dv, alias):
    """Two keys a row whose values are each other's opposites and whose scores differ by about 2^-13: what is left of the output is the difference
    of two weights near 1, which a weight of 16 bits (2^-17 off) gives to one or two digits only."""
    g = torch.Generator(device="cuda")
    g.manual_seed(dk)
    L = 200
    k = torch.zeros(1, L, dk, dtype=torch.bfloat16, device="cuda")
    tail = dv if alias else 0                                                # (the entries that the queries look at)
    k[0, :, tail] = 0.25
    k[0, :, tail + 1] = (torch.rand(L, generator=g, device="cuda") * 2.0 ** -12).bfloat16()
    v = ((torch.rand(dv, generator=g, device="cuda") + 0.5) * (1.0 - 2.0 * (torch.arange(L, device="cuda") % 2))[:, None]).bfloat16()
    if alias:
        k[0, :, :dv] = v
    q = torch.zeros(L, H, dk, dtype=torch.bfloat16, device="cuda")
    q[:, :, tail] = torch.rand(L, H, generator=g, device="cuda").bfloat16()
    q[:, :, tail + 1] = 1.0
    kp, vp, table = paged(k, None if alias else v[None])
    out = torch.full((L, H * dv), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops = Ops(torch.bfloat16)
    assert lib("attention_scored_prompt").kvad_attention_scored_prompt_takes(dk, dv, int(alias), 0) == 1
    ops.attention_scored(q.view(L, -1), out, i32([0, L]), i32([L]), 1, L, table, kp, vp, H, 1.0, value_dim=dv if alias else None, window=2)
    x = torch.einsum("thd,sd->hts", q.double(), k[0].double())
    pos = torch.arange(L, device="cuda")
    x = x.masked_fill((pos[None] > pos[:, None]) | (pos[None] <= pos[:, None] - 2), float("-inf"))
    want = torch.einsum("hts,sd->thd", torch.softmax(x, 2), v.double()).reshape(L, -1)
    # scores of at most 1/4 + 2^-12, rounded a few times: 2^-24 of a weight; an exponential good to 2 units in the last place: 2^-23; the output's own rounding
    bound = 2.0 ** -8 * want.abs() + 2.0 ** -21 * v.double().abs().max(0).values.repeat(H)
    assert ((out.double() - want).abs() <= bound).all(), ((out.double() - want).abs() / bound).max().item()


@pytest.mark.parametrize("H,dk,dv,alias,cached", [(16, 64, 64, False, 16384), (16, 128, 128, True, 8192), (16, 256, 256, True, 8192)])
def test_a_long_cache_adds_no_bias(H, dk, dv, alias, cached):
    """Positive values under nearly even weights: a sum that truncates at every step falls behind the longer it gets.  The outputs' own roundings, spread by a
    gate, average out over the rows."""
    g = torch.Generator(device="cuda")
    g.manual_seed(dv)
    new = 256
    L = cached + new
    k = (torch.rand(1, L, dk, generator=g, device="cuda") + 0.5).bfloat16()
    v = None if alias else (torch.rand(1, L, dv, generator=g, device="cuda") + 0.5).bfloat16()
    q, gate = (torch.randn(new, H * d, generator=g, device="cuda").bfloat16() for d in (dk, dv))
    kp, vp, table = paged(k, v)
    out = torch.full((new, H * dv), float("nan"), dtype=torch.bfloat16, device="cuda")
    scale = 0.1 / dk ** 0.5
    Ops(torch.bfloat16).attention_scored(q, out, i32([0, new]), i32([L]), 1, new, table, kp, vp, H, scale, value_dim=dv if alias else None, gate=gate)
    seen = torch.arange(L, device="cuda")[None] <= torch.arange(cached, L, device="cuda")[:, None]
    vd = (k if alias else v)[0, :, :dv].double()
    error = 0.0
    for h in range(H):
        x = (q[:, h * dk:(h + 1) * dk].double() @ k[0].double().t() * scale).masked_fill(~seen, float("-inf"))
        want = torch.softmax(x, 1) @ vd * torch.sigmoid(gate[:, h * dv:(h + 1) * dv].double())
        error += ((out[:, h * dv:(h + 1) * dv].double() - want) / want).mean().item() / H
    # single roundings to bfloat16 are 2^-9 at most and of either sign: 256 rows of 1024 outputs or more leave 2^-9 / 2^9 / sqrt(3) of them, four times that
    # is 2^-16.8; 32-bit sums by rounding are far below
    assert abs(error) < 2.0 ** -17, error


@pytest.mark.parametrize("cap", [0.5, 5.0, 30.0, 1000.0, 1e6, 3e38])
@pytest.mark.parametrize("H,G,dk,dv,form", [(4, 2, 64, 64, {}), (16, 1, 128, 128, dict(alias=True, sinks=True)), (4, 4, 256, 256, dict(window=90))])
def test_score_caps_of_any_size(H, G, dk, dv, form, cap):
    """The error of a capped score follows the score, not the cap: prompts and single-token rows, 16-bit and 32-bit outputs."""
    ops = Ops(torch.bfloat16)
    for seqs in (EDGES, STEPS):
        c = Case(seqs, H, G, dk, dv, cap=cap, **form)
        for out in (torch.bfloat16, torch.float32):
            c.check(c.run(ops, out), out)


def test_a_prompt_of_more_tiles_than_a_grid_dimension_holds():
    """16 heads on one key make tiles of 4 tokens: from 262 141 rows on there are more than 65 535 of them."""
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    new, H, dk = 65535 * 4 + 70, 16, 8
    L = new + 5
    k = torch.randn(1, L, dk, generator=g, device="cuda").bfloat16()
    q = torch.randn(new, H * dk, generator=g, device="cuda").bfloat16()
    kp, _, table = paged(k, None)
    out = torch.full((new, H * dk), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops = Ops(torch.bfloat16)
    kw = dict(value_dim=dk, window=40)
    ops.attention_scored(q, out, i32([0, new]), i32([L]), 1, new, table, kp, None, H, 0.3, **kw)
    cut = new - 3000
    part = torch.full((3000, H * dk), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.attention_scored(q[cut:], part, i32([0, 3000]), i32([L]), 1, 3000, table, kp, None, H, 0.3, **kw)
    assert torch.equal(out[cut:], part)
    first = torch.full((3000, H * dk), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.attention_scored(q[:3000], first, i32([0, 3000]), i32([3005]), 1, 3000, table, kp, None, H, 0.3, **kw)
    assert torch.equal(out[:3000], first) and out.isfinite().all()


# tiles of 128 (token, head) pairs, products of 64 and 128 columns, one to four pages on their way; caps whose scores lie on both sides of the polynomial's range
TILES = [
    (4, 4, 64, 64, dict(cap=3.0)), (4, 4, 64, 64, dict(cap=300.0, gate="entry")), (2, 2, 128, 128, {}), (8, 1, 80, 72, {}), (8, 1, 136, 136, dict(window=64, keep=65)),
    (16, 2, 200, 200, dict(sinks=True)), (16, 1, 288, 256, dict(alias=True)), (16, 1, 576, 256, dict(alias=True, chunk=64)), (2, 1, 384, 128, dict(span=8.0)), (32, 1, 64, 192, {}),
]


@pytest.mark.parametrize("H,G,dk,dv,form", TILES)
def test_prompt_tiles(H, G, dk, dv, form):
    from kvad_b200.ops import scored_prompt_wait_timeouts
    assert lib("attention_scored_prompt").kvad_attention_scored_prompt_takes(dk, dv, int("alias" in form), 0) == 1
    c = Case([(0, 128), (64, 64), (0, 257), (449, 31), (3, 2), (0, 1)], H, G, dk, dv, **form)
    for out in [torch.bfloat16] if c.gate is not None else [torch.bfloat16, torch.float32]:
        c.check(c.run(Ops(torch.bfloat16), out), out)
    assert scored_prompt_wait_timeouts() == 0


def rows_by_formula(c, s=0):
    """The rows of sequence `s` in 64 bits, each from the keys and values that it sees and nothing else."""
    cached, new = c.seqs[s]
    kw, H, L = c.kw, c.H, cached + new
    first = int(c.starts[s])
    take = lambda p, width: p[c.table[s].long()].double().permute(1, 0, 2, 3).reshape(p.shape[1], -1, p.shape[3])[:, :L, :width]
    k = take(c.kp, c.kp.shape[3])
    v = (k[:, :, :c.dv] if c.vp is None else take(c.vp, c.dv)).repeat_interleave(kw["key_maps"], 0)
    k, v = k.repeat_interleave(H // k.shape[0], 0), v.repeat_interleave(H // v.shape[0], 0)
    q = c.q[first:first + new].double().reshape(new, H, -1)
    out = torch.empty(new, H, c.dv, dtype=torch.float64, device="cuda")
    for i in range(new):
        pos, key = cached + i, torch.arange(cached + i + 1, device="cuda")
        seen = torch.ones_like(key, dtype=torch.bool)
        if kw["window"]:
            seen = (key > pos - kw["window"]) | (key < kw["keep_first"])
        if kw["chunk"]:
            seen = key >= pos - pos % kw["chunk"]
        at = key[seen]
        x = (k[:, at] * q[i][:, None, :]).sum(2) * c.scale
        if kw["softcap"]:
            x = kw["softcap"] * torch.tanh(x / kw["softcap"])
        if kw["slope_span"]:
            x = x - (2.0 ** (-kw["slope_span"] * torch.arange(1, H + 1, device="cuda").double() / H))[:, None] * (pos - at)[None]
        if c.sinks is not None:
            x = torch.cat([x, c.sinks.double()[:, None]], 1)
        o = (torch.softmax(x, 1)[:, :len(at), None] * v[:, at]).sum(1)
        if c.gate is not None:
            o = o * torch.sigmoid(c.gate[first + i].double().reshape(H, -1))
        out[i] = o
    return out.reshape(new, -1)


# the number lies at position 104 of the first sequence: in the middle of a tile, and (one head a group) of a page that other tiles' rows end in
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("where", ["q", "k", "v"])
@pytest.mark.parametrize("H,G,dk,dv,form", [
    (4, 4, 64, 64, {}), (16, 1, 64, 64, dict(span=8.0)), (8, 2, 128, 128, dict(window=20, keep=4, gate="entry")), (16, 1, 256, 256, dict(alias=True, gate="head")),
    (4, 2, 200, 200, dict(sinks=True)), (2, 1, 72, 136, dict(chunk=96, cap=5.0)), (8, 8, 64, 64, dict(key_maps=2, window=40))])
def test_a_number_that_is_not_finite_stays_with_the_rows_that_see_it(H, G, dk, dv, form, where, bad):
    c = Case([(70, 150), (3, 40)], H, G, dk, dv, **form)
    if where == "q":
        c.q[34, dk + 5] = bad                             # head 1 of position 104
    else:
        (c.kp if where == "k" or c.vp is None else c.vp)[c.table[0, 1].long(), 0, 40, 5] = bad
    want = c.want.clone()
    want[:150] = rows_by_formula(c)
    assert want[150:].isfinite().all() and (not want[:150].isfinite().all() or (where != "v" and bad == float("inf")))      # (a score of minus infinity hides a key, a cap makes it finite)
    for out in [torch.bfloat16] if c.gate is not None else [torch.bfloat16, torch.float32]:
        got = c.run(Ops(torch.bfloat16), out)
        assert torch.equal(got.isfinite(), want.isfinite())
        ok = want.isfinite()
        # (a row that loses a key's weight keeps its bound's order: twice it is generous)
        bound = 2 * c.slack + (2.0 ** -8 if out == torch.bfloat16 else 2.0 ** -22) * want.abs() + 1e-30
        assert float(((got - want).abs() / bound)[ok].max()) <= 1.0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_a_capped_rows_bits_are_its_own(dtype):
    """Scores far out, where the cap takes another formula, in later rows of the tile, in another sequence and in places of the cache that hold nothing yet."""
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    ops, H, G, d = Ops(dtype), 4, 2, 64
    kp, vp, q = (torch.randn(*s, generator=g, device="cuda").to(dtype) for s in ((5, G, PAGE, d), (5, G, PAGE, d), (50, H * d)))
    table = i32([[3, 1], [0, 4]])

    def run(q, kp, n_seqs):
        out = torch.full((50 if n_seqs == 2 else 20, H * d), float("nan"), device="cuda")      # (32-bit: a rounding to 16 would hide it)
        ops.attention_scored(q[:len(out)], out, i32([0, 20, 50][:n_seqs + 1]), i32([90, 35][:n_seqs]), n_seqs, 30 if n_seqs == 2 else 20, table[:n_seqs], kp, vp, H, 0.125, softcap=30.0)
        return out
    want = run(q, kp, 1)
    assert want.isfinite().all()
    far = q.clone()
    far[10:] *= 1000
    assert torch.equal(run(far, kp, 1)[:10], want[:10])
    far = q.clone()
    far[20:] *= 1000
    assert torch.equal(run(far, kp, 2)[:20], want)
    stale = kp.clone()
    stale[1, :, 90 - PAGE:] *= 1000                      # places past the first sequence's end
    assert torch.equal(run(q, stale, 1), want)


@pytest.mark.parametrize("H,G,dk,dv", [(4, 2, 64, 64), (16, 1, 256, 256)])
@pytest.mark.parametrize("gate", ["entry", "head"])
def test_gates_far_below_zero(H, G, dk, dv, gate):
    """sigmoid(-88) is 6e-39: 1 + e^88 lies where a fast division gives 0."""
    c = Case([(3, 70)], H, G, dk, dv, gate=gate)
    f = torch.sigmoid(c.gate.double())
    c.gate.fill_(-88.0)
    c.vp.mul_(2.0 ** 100)
    wide = (lambda x: x.repeat_interleave(dv, 1)) if gate == "head" else (lambda x: x)
    change = wide(torch.sigmoid(c.gate.double()) / f) * 2.0 ** 100
    got, want, slack = c.run(Ops(torch.bfloat16)), c.want * change, c.slack * change
    assert ((got - want).abs() <= slack + 2.0 ** -8 * want.abs() + 1e-30).all()
    assert float(want.abs().max()) > 1e-9


@pytest.mark.parametrize("H,G,dk,dv,form", [(8, 2, 520, 64, {}), (4, 1, 528, 8, dict(cap=3.0, sinks=True)), (2, 2, 576, 256, dict(window=70, keep=65)), (4, 2, 512, 256, dict(gate="entry")),
                                            (4, 1, 528, 72, dict(chunk=96))])
def test_keys_so_long_that_keys_and_values_of_a_page_come_in_turn(H, G, dk, dv, form):
    from kvad_b200.ops import scored_prompt_wait_timeouts
    assert lib("attention_scored_prompt").kvad_attention_scored_prompt_takes(dk, dv, 0, 0) == 1
    c = Case([(0, 128), (64, 64), (449, 31), (3, 2), (0, 1)], H, G, dk, dv, **form)
    for out in [torch.bfloat16] if c.gate is not None else [torch.bfloat16, torch.float32]:
        c.check(c.run(Ops(torch.bfloat16), out), out)
    assert scored_prompt_wait_timeouts() == 0
