"""32-bit prompt attention with shaped scores on the tensor cores (operands in bfloat16 pieces) against the formula in 64 bits and the CUDA-core kernel: ends of
tiles and pages, every shaping of a score, sizes that fill no 16 or 64, pages with no number where no row lies, numbers that are not finite."""
import pytest
import torch

from kvad_b200.ops import Ops, lib, scored_wide_wait_timeouts
from tests.test_gpu_scored_forms import rows_by_formula

pytestmark = pytest.mark.gpu
PAGE = 64


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


class Case:
    def __init__(self, seqs, H, G, dk, dv, *, alias=False, key_maps=1, cap=0.0, span=0.0, window=0, keep=0, chunk=0, gate=None, sinks=False):
        g = torch.Generator(device="cuda")
        g.manual_seed(dk * 7 + dv + H)
        rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
        self.seqs, self.H, self.scale, self.key_maps = seqs, H, 1.5 / dk ** 0.5, key_maps
        self.cap, self.span, self.window, self.keep, self.chunk = cap, span, window, keep, chunk
        self.kw = dict(softcap=cap, slope_span=span, window=window, keep_first=keep, chunk=chunk, key_maps=key_maps)
        width = -(-max(c + n for c, n in seqs) // PAGE)
        order = torch.randperm(width * len(seqs) + 2, generator=torch.Generator().manual_seed(3))
        self.table = order[:width * len(seqs)].reshape(len(seqs), width).to(torch.int32).cuda().contiguous()
        self.kp = torch.full((len(order), G, PAGE, dk), float("nan"), device="cuda")
        self.vp = None if alias else torch.full((len(order), G // key_maps, PAGE, dv), float("nan"), device="cuda")
        n_rows = sum(n for _, n in seqs)
        self.q = rnd(n_rows, H * dk + 4)[:, :H * dk]
        self.gate = {None: None, "entry": rnd(n_rows, H * dv), "head": rnd(n_rows, H)}[gate]
        self.sinks = rnd(H) if sinks else None
        self.dv, self.out = dv, (n_rows, H * dv)
        for s, (cached, new) in enumerate(seqs):
            for j in range(cached + new):
                self.kp[self.table[s, j // PAGE].long(), :, j % PAGE] = rnd(G, dk)
                if not alias:
                    self.vp[self.table[s, j // PAGE].long(), :, j % PAGE] = rnd(G // key_maps, dv)
        starts = [0]
        for _, n in seqs:
            starts.append(starts[-1] + n)
        self.starts, self.lens, self.max_new = i32(starts), i32([c + n for c, n in seqs]), max(n for _, n in seqs)

    def want(self):
        outs, at, H = [], 0, self.H
        for s, (cached, new) in enumerate(self.seqs):
            L = cached + new
            pages = self.table[s, :-(-L // PAGE)].long()
            rows = lambda p: p[pages].double().permute(1, 0, 2, 3).reshape(p.shape[1], -1, p.shape[3])[:, :L]
            k = rows(self.kp)
            v = k[..., :self.dv] if self.vp is None else rows(self.vp).repeat_interleave(self.key_maps, 0)
            k, v = k.repeat_interleave(H // k.shape[0], 0), v.repeat_interleave(H // v.shape[0], 0)
            x = self.q[at:at + new].double().reshape(new, H, -1).transpose(0, 1) @ k.transpose(1, 2) * self.scale
            if self.cap:
                x = self.cap * torch.tanh(x / self.cap)
            pos, key = torch.arange(cached, L, device="cuda"), torch.arange(L, device="cuda")
            if self.span:
                x = x - (2.0 ** (-self.span * torch.arange(1, H + 1, device="cuda").double() / H))[:, None, None] * (pos[:, None] - key[None, :])
            seen = key[None, :] <= pos[:, None]
            if self.window:
                seen &= (key[None, :] > pos[:, None] - self.window) | (key[None, :] < self.keep)
            if self.chunk:
                seen &= key[None, :] >= (pos - pos % self.chunk)[:, None]
            x = x.masked_fill(~seen, float("-inf"))
            if self.sinks is not None:
                x = torch.cat([x, self.sinks.double()[:, None, None].expand(H, new, 1)], 2)
            o = torch.softmax(x, 2)[:, :, :L] @ v
            if self.gate is not None:
                o = o * torch.sigmoid(self.gate[at:at + new].double().reshape(new, H, -1)).transpose(0, 1)
            outs.append(o.transpose(0, 1).reshape(new, -1))
            at += new
        return torch.cat(outs)

    def run(self, ops):
        out = torch.full((self.out[0], self.out[1] + 4), float("nan"), device="cuda")
        ops.attention_scored(self.q, out[:, :-4], self.starts, self.lens, len(self.seqs), self.max_new, self.table, self.kp, self.vp, self.H, self.scale,
                             value_dim=self.dv, softcap=self.cap, slope_span=self.span, window=self.window, keep_first=self.keep, chunk=self.chunk,
                             key_maps=self.key_maps, sinks=self.sinks, gate=self.gate)
        torch.cuda.synchronize()
        assert out[:, -4:].isnan().all()
        return out[:, :-4].double()


EDGES = [(0, 129), (63, 2), (200, 65), (5, 1), (0, 64), (1, 127), (449, 31)]
FORMS = [
    (4, 4, 64, 64, {}), (16, 4, 64, 64, dict(cap=30.0, window=100, keep=4, gate="entry")), (8, 2, 128, 128, dict(gate="head")), (6, 2, 72, 40, dict(cap=3.0)),
    (16, 1, 96, 64, dict(alias=True, sinks=True)), (4, 2, 32, 32, dict(chunk=96)), (8, 8, 64, 64, dict(key_maps=2)), (4, 2, 128, 64, dict(span=8.0)),
    (8, 1, 160, 128, dict(alias=True)), (2, 1, 8, 8, dict(sinks=True, window=130, keep=70, cap=5.0, span=4.0)), (20, 1, 64, 24, dict(window=1)),
]


@pytest.mark.parametrize("H,G,dk,dv,form", FORMS)
def test_no_further_off_than_the_cuda_cores(H, G, dk, dv, form):
    assert lib("attention_scored_wide").kvad_attention_scored_wide_takes(dk, dv, int("alias" in form)) == 1
    c, ops, cores = Case(EDGES, H, G, dk, dv, **form), Ops(torch.float32), Ops(torch.float32)
    cores.scored_wide = False
    want = c.want()
    far = [float((c.run(o) - want).norm() / want.norm()) for o in (ops, cores)]
    # six products leave out 2^-23 of a score's terms, scores of up to 2^4 pass that on to the weights; the rest is what the cores' chains lose too
    assert far[0] < max(1.2 * far[1], 4e-7), far
    assert scored_wide_wait_timeouts() == 0


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("where", ["q", "k", "v"])
def test_numbers_that_are_not_finite(where, bad):
    """Rows that see the number, of the heads that read it, are not finite (the CUDA cores' rows that see its page neither); the others are what they are there."""
    c = Case([(70, 130), (3, 40)], 4, 2, 64, 64)
    if where == "q":
        c.q[20, 70] = bad                                 # head 1 of one row
        see, others = [(slice(20, 21), slice(64, 128))], (slice(0, 20), slice(0, 256))
    else:
        (c.kp if where == "k" else c.vp)[c.table[0, 1].long(), 1, 40, 5] = bad          # position 104, read by heads 2 and 3
        cols = [slice(128, 256)] if where == "k" else [slice(133, 134), slice(197, 198)]
        see, others = [(slice(34, 130), x) for x in cols], (slice(0, 34), slice(0, 256))
    ops, cores = Ops(torch.float32), Ops(torch.float32)
    cores.scored_wide = False
    got, want = c.run(ops), c.run(cores)
    for rows, cols in see:
        assert not got[rows, cols].isfinite().any() or (where == "k" and bad == float("inf"))      # (a score of minus infinity hides the key)
    assert got[others].isfinite().all() and (got.isfinite() | ~want.isfinite()).all()
    ok = want.isfinite()
    assert float((got[ok] - want[ok]).abs().max()) < 2e-6


# position 104 of the first sequence: in the middle of a tile, and (one head a group) of a page that other tiles' rows end in
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("where", ["q", "k", "v"])
@pytest.mark.parametrize("H,G,dk,dv,form", [(4, 4, 64, 64, {}), (16, 1, 96, 64, dict(alias=True, sinks=True)), (8, 2, 128, 128, dict(window=20, keep=4, gate="entry")),
                                            (6, 2, 72, 40, dict(cap=3.0)), (8, 8, 64, 64, dict(key_maps=2, chunk=40, gate="head"))])
def test_a_number_that_is_not_finite_stays_with_the_rows_that_see_it(H, G, dk, dv, form, where, bad):
    c = Case([(70, 150), (3, 40)], H, G, dk, dv, **form)
    clean = c.want()
    if where == "q":
        c.q[34, dk + 5] = bad                             # head 1 of position 104
    else:
        (c.kp if where == "k" or c.vp is None else c.vp)[c.table[0, 1].long(), 0, 40, 5] = bad
    want = torch.cat([rows_by_formula(c), clean[150:]])
    assert want[150:].isfinite().all() and (not want[:150].isfinite().all() or (where != "v" and bad == float("inf")))      # (a score of minus infinity hides a key, a cap makes it finite)
    got = c.run(Ops(torch.float32))
    assert torch.equal(got.isfinite(), want.isfinite())
    ok = want.isfinite()
    assert float((got - want)[ok].abs().max()) < 1e-5      # (scores of up to 2^4 with errors of 2^-21: a weight's of 2^-17)
    assert scored_wide_wait_timeouts() == 0


@pytest.mark.parametrize("scale", [0.01, 0.3])
@pytest.mark.parametrize("H,G,dk,dv,alias", [(4, 2, 64, 64, False), (4, 1, 160, 128, True), (4, 2, 128, 128, False)])
def test_numbers_of_one_sign(H, G, dk, dv, alias, scale):
    """Sums to which every term adds, where an accumulator that truncates falls behind: no further off than the CUDA cores' chains of fmaf, from one page to many."""
    ops, cores = Ops(torch.float32), Ops(torch.float32)
    cores.scored_wide = False
    for seqs in ([(0, 17), (3, 70)], [(0, 300)], [(1500, 60)]):
        c = Case(seqs, H, G, dk, dv, alias=alias, sinks=True)
        c.q, c.kp, c.scale, c.sinks = c.q.abs(), c.kp.abs(), scale / dk ** 0.5, c.sinks + scale * dk ** 0.5 * 2 / 3.14
        c.vp = None if alias else c.vp.abs()
        want = c.want()
        far, bias = zip(*[(float((x - want).norm() / want.norm()), float(((x - want) / want).mean())) for x in (c.run(ops), c.run(cores))])
        # 2^-23: exponentials good to 2 units in the last place; a page's sums truncate at their last four steps, 2^-25 of the sum each on the average
        assert far[0] < max(1.1 * far[1], 2.0 ** -23) and abs(bias[0]) < 2.0 ** -23, (far, bias)


@pytest.mark.parametrize("H,d,window", [(12, 64, 0), (12, 64, 20), (25, 32, 0)])
def test_short_prompts_beside_longer_ones(H, d, window):
    """More blocks than SMs: sequences of a page at most go to the CUDA cores, the others to the tensor cores; no place is left out or written twice."""
    ops, cores = Ops(torch.float32), Ops(torch.float32)
    cores.scored_wide = False
    c = Case([(0, 32), (60, 4), (61, 4), (0, 1), (33, 31), (33, 32), (200, 20)] * 4, H, H, d, d)      # (of 32 new rows at most)
    outs = []
    for o in (ops, cores):
        out = torch.full((c.out[0], H * d), float("nan"), device="cuda")
        o.attention_prompt(c.q, out, c.starts, c.lens, len(c.seqs), c.max_new, c.table, c.kp, c.vp, H, c.scale, window)
        outs.append(out)
    assert outs[0].isfinite().all() and float((outs[0] - outs[1]).abs().max()) < 1e-5
    at = 0
    for cached, new in c.seqs:                           # (the same kernel: the same bits; another: not)
        same = torch.equal(outs[0][at:at + new], outs[1][at:at + new])
        assert same == (cached + new <= 64) or new == 1
        at += new
