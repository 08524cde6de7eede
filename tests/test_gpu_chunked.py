"""Recurrences of prompts taken in chunks of 64 rows, against the row by row formulas in 64 bits: ragged lengths around the edges of chunks
and blocks, states carried on, sizes that fill no tile, decays of 0 and 1."""
import numpy as np
import pytest
import torch

from kvad_b200.ops import Ops, lib

pytestmark = pytest.mark.gpu
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}
LENS = [65, 1, 129, 64, 300, 16, 63]
SLOTS = [6, 0, 3, 8, 1, 5, 2]                 # slots 4 and 7 belong to nobody


def rel(got, ref):
    return float((got.double() - ref).norm() / ref.norm().clamp(min=1e-30))


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device="cuda")


def starts(lens):
    return i32([0] + list(np.cumsum(lens)))


def portions():
    """All rows at once; and in two steps, the second of which carries the first one's state on."""
    yield [LENS]
    yield [[min(n, 70) for n in LENS], [n - min(n, 70) for n in LENS]]


def rows(x, lens, done, part):
    at = np.cumsum([0] + lens[:-1])
    return torch.cat([x[a + d:a + d + p] for a, d, p in zip(at, done, part)])


def walk(lens, H, dk, dv, q, k, v, g, beta=None, w=None):
    """S = g S + w k u^T row by row; `g` [n, H, dk] or [n, H, 1].  Read-outs and the states at the ends."""
    outs, ends, at = [], [], 0
    for n in lens:
        S = torch.zeros(H, dk, dv, dtype=torch.float64, device="cuda")
        for t in range(at, at + n):
            S = S * g[t][:, :, None]
            u = v[t] if beta is None else beta[t][:, None] * (v[t] - (S * k[t][:, :, None]).sum(1))
            S = S + (k[t] if w is None else k[t] * w[t][:, None])[:, :, None] * u[:, None, :]
            outs.append((S * q[t][:, :, None]).sum(1))
        ends.append(S)
        at += n
    return torch.stack(outs), ends


def through(call, lens, out_width):
    """The rows in the given portions through `call(select, starts, slots, lens after, n, out)`; read-outs of all rows in their order."""
    got = []
    for cuts in portions():
        out = torch.full((sum(lens), out_width), float("nan"), device="cuda")
        state, done, at = None, [0] * len(lens), np.cumsum([0] + lens[:-1])
        for part in cuts:
            live = [i for i in range(len(lens)) if part[i]]
            o = torch.full((sum(part), out_width), float("nan"), device="cuda")
            after = [done[i] + part[i] for i in live]
            state = call(lambda x: rows(x, lens, done, part), starts([part[i] for i in live]), i32([SLOTS[i] for i in live]), i32(after), len(live), o, state)
            pos = 0
            for i in live:
                out[at[i] + done[i]:at[i] + done[i] + part[i]] = o[pos:pos + part[i]]
                pos += part[i]
            done = [d + p for d, p in zip(done, part)]
        got.append((out, state))
    return got


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,dk,dv,rot,inter,act", [(2, 128, 128, 128, False, False), (3, 64, 20, 0, False, True), (1, 4, 64, 4, True, False), (2, 100, 68, 32, False, False)])
def test_retention_in_chunks(dtype, H, dk, dv, rot, inter, act):
    g, ops = torch.Generator(device="cuda"), Ops(DT[dtype])
    g.manual_seed(dk + dv)
    ops.CHUNK_MIN_ROWS = 1
    N, t = sum(LENS), DT[dtype]
    q, k, v, gate = (torch.randn(N, H * d, generator=g, device="cuda").to(t) for d in (dk, dk, dv, dv))
    decay = torch.linspace(0.9, 1.0, H, device="cuda") if H > 1 else torch.tensor([0.97], device="cuda")
    freq = (100.0 ** (-torch.arange(0, max(rot, 2), 2, device="cuda") / max(rot, 2))).float() if rot else None
    ks, eps = dk ** -0.5, 1e-5
    s = torch.nn.functional.silu if act else (lambda x: x)
    qd, kd, vd = (s(x.double()).view(N, H, -1).clone() for x in (q, k, v))
    pos = torch.cat([torch.arange(n, device="cuda") for n in LENS]).double()
    if rot:
        ang = (pos[:, None].float() * freq).double()[:, None, :]          # angles as the kernel has them, in 32 bits
        c, sn = torch.cos(ang), torch.sin(ang)
        for x in (qd, kd):
            a, b = (x[..., 0:rot:2], x[..., 1:rot:2]) if inter else (x[..., :rot // 2], x[..., rot // 2:rot])
            a1, b1 = a * c - b * sn, b * c + a * sn
            if inter:
                x[..., 0:rot:2], x[..., 1:rot:2] = a1, b1
            else:
                x[..., :rot // 2], x[..., rot // 2:rot] = a1, b1
    raw, ends = walk(LENS, H, dk, dv, qd, kd * ks, vd, decay.double()[None, :, None].expand(N, H, 1))
    kw = dict(inv_freq=freq, rot_dims=rot, interleaved=inter, k_scale=ks, silu_inputs=act)

    def run(finish):
        def call(pick, st, sl, after, n, out, state):
            state = torch.zeros(9, H, dk, dv, device="cuda") if state is None else state
            if finish:
                o = torch.full(out.shape, float("nan"), device="cuda", dtype=t)
                scratch = torch.empty(out.shape, device="cuda")
                ops.retention(pick(q), pick(k), pick(v), o, state, st, after, sl, n, decay, H, gate=pick(gate), unit_norm_eps=eps, raw=scratch, **kw)
                out.copy_(o)
            else:
                ops.retention(pick(q), pick(k), pick(v), None, state, st, after, sl, n, decay, H, raw=out, raw_only=True, **kw)
            return state
        return through(call, LENS, H * dv)

    gd = gate.double().view(N, H, dv)
    done = raw / torch.sqrt(raw.square().mean(-1, keepdim=True) + eps) * gd * torch.sigmoid(gd)
    for finish, want in ((False, raw), (True, done)):
        for out, state in run(finish):
            # 32-bit sums of up to 192 terms a chunk; 32-bit sines; the finished rows of bfloat16 are rounded once
            assert rel(out.view(N, H, dv), want) < (5e-3 if finish and dtype == "bfloat16" else 3e-6)
            assert all(rel(state[SLOTS[i]], e) < 3e-6 for i, e in enumerate(ends)) and float(state[[4, 7]].abs().max()) == 0.0


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,G,dk,dv", [(2, 2, 128, 128), (4, 2, 64, 20), (1, 1, 4, 64), (3, 1, 100, 72)])
def test_matrix_memory_in_chunks(dtype, H, G, dk, dv):
    g, ops, cap = torch.Generator(device="cuda"), Ops(DT[dtype]), 15.0
    g.manual_seed(dk + dv)
    ops.CHUNK_MIN_ROWS = 1
    N, t, tiles = sum(LENS), DT[dtype], -(-dv // 16)
    q, k, v = (torch.randn(N, n * d, generator=g, device="cuda").to(t) for n, d in ((G, dk), (G, dk), (H, dv)))
    gates = torch.randn(N, 2 * H, generator=g, device="cuda") * 3.0
    gates[:, H:] += 4.0
    gates[200:230, H:] -= 200.0                # a stretch that forgets at the cap: sums of logarithms in the hundreds
    scale = dk ** -0.5
    qd, kd, vd = (x.double().view(N, -1, d).repeat_interleave(r, 1) for x, d, r in ((q, dk, H // G), (k, dk, H // G), (v, dv, 1)))
    gi, gf = cap * torch.tanh(gates[:, :H].double() / cap), torch.nn.functional.logsigmoid(cap * torch.tanh(gates[:, H:].double() / cap))
    m, f, w = (torch.empty(N, H, dtype=torch.float64, device="cuda") for _ in range(3))
    at = 0
    for n in LENS:
        last = torch.zeros(H, dtype=torch.float64, device="cuda")
        for r in range(at, at + n):
            m[r] = torch.maximum(gf[r] + last, gi[r])
            f[r], w[r] = torch.exp(gf[r] + last - m[r]), torch.exp(gi[r] - m[r])
            last = m[r]
        at += n
    one = torch.ones(N, H, 1, dtype=torch.float64, device="cuda")
    num, ends = walk(LENS, H, dk, dv, qd * scale, kd, vd, f[:, :, None], w=w)
    den, n_ends = walk(LENS, H, dk, 1, qd * scale, kd, one, f[:, :, None], w=w)
    want = num / (torch.maximum(den.abs(), torch.exp(-m)[:, :, None]) + 1e-6)

    def call(pick, st, sl, after, n, out, state):
        state = torch.zeros(9, ops.recurrence_state_size("matrix_memory", H, dk, dv), device="cuda") if state is None else state
        state = torch.nn.functional.pad(state, (0, -state.shape[1] % 4)) if state.shape[1] % 4 else state
        ops.gated_recurrence("matrix_memory", pick(q), pick(k), pick(v), pick(gates), out, state, st, sl, n, H, G, dk, dv, q_scale=scale, cap=cap)
        return state

    # The gates' logarithms are 32-bit numbers whose errors add up over a reach of rows, in either kernel: a logarithm of up to 15 is off by
    # 2^-21, and a memory reaches back at most 129 rows that such errors do not cancel over: sqrt(129) 2^-21 times three.
    tol = 3.0 * 129 ** 0.5 * 2.0 ** -21
    for out, state in through(call, LENS, H * dv):
        # a quotient whose sums can nearly cancel
        assert rel(out.view(N, H, dv), want) < 5e-5
        last = np.cumsum(LENS) - 1
        for i, (e, ne) in enumerate(zip(ends, n_ends)):
            st = state[SLOTS[i]]
            assert rel(st[:H * dv * dk].view(H, dv, dk).transpose(1, 2), e) < tol
            norms = st[H * dv * dk:H * dv * dk + H * tiles * dk].view(H, tiles, dk)
            assert all(rel(norms[:, j], ne[..., 0]) < tol for j in range(tiles))
            maxima = st[H * dv * dk + H * tiles * dk:H * dv * dk + H * tiles * (dk + 1)].view(H, tiles).double()
            assert torch.allclose(maxima, m[last[i]][:, None].expand(-1, tiles), rtol=tol, atol=tol)
        assert float(state[[4, 7]].abs().max()) == 0.0


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("kind", ["delta_rule", "gated_linear"])
@pytest.mark.parametrize("H,G,dk,dv", [(2, 2, 128, 128), (4, 2, 64, 20), (1, 1, 4, 64), (3, 1, 100, 72), (2, 1, 36, 7)])
def test_channel_recurrences_in_chunks(dtype, kind, H, G, dk, dv):
    g, ops = torch.Generator(device="cuda"), Ops(DT[dtype])
    g.manual_seed(dk + dv)
    ops.CHUNK_MIN_ROWS = 1
    N, t, delta = sum(LENS), DT[dtype], kind == "delta_rule"
    q, k, v = (torch.randn(N, n, d, generator=g, device="cuda") for n, d in ((G, dk), (G, dk), (H, dv)))
    if delta:
        k = torch.nn.functional.normalize(k, dim=-1)
        k[40:60] = k[40]                          # one key again and again: what was written is taken back every time
    q, k, v = q.reshape(N, -1).to(t), k.reshape(N, -1).to(t), v.reshape(N, -1).to(t)
    decay = torch.sigmoid(torch.randn(N, H, dk, generator=g, device="cuda") + 2.0)
    decay[:, :, 0], decay[:, :, 1] = 1.0, 0.0     # a channel that keeps everything, one that keeps nothing
    decay[100:103, :, 2] = 1e-30                  # products of these underflow
    beta = torch.sigmoid(torch.randn(N, H, generator=g, device="cuda"))
    scale = 0.5
    qd, kd = (x.double().view(N, G, dk).repeat_interleave(H // G, 1) for x in (q, k))
    want, ends = walk(LENS, H, dk, dv, qd * scale, kd, v.double().view(N, H, dv), decay.double(), beta=beta.double() if delta else None)
    more = dict(beta=beta, a_log=torch.zeros(H, device="cuda"), dt_bias=torch.zeros(H * dk, device="cuda")) if delta else {}

    def call(pick, st, sl, after, n, out, state):
        state = torch.zeros(9, ops.recurrence_state_size(kind, H, dk, dv) + 3, device="cuda") if state is None else state
        kw = dict(more, beta=pick(beta)) if delta else {}
        ops.gated_recurrence(kind, pick(q), pick(k), pick(v), pick(decay.view(N, -1)), out, state, st, sl, n, H, G, dk, dv, q_scale=scale, gates_ready=True, **kw)
        return state

    for out, state in through(call, LENS, H * dv):
        assert rel(out.view(N, H, dv), want) < 3e-6
        for i, e in enumerate(ends):
            assert rel(state[SLOTS[i]][:H * dv * dk].view(H, dv, dk).transpose(1, 2), e) < 3e-6
        assert float(state[[4, 7]].abs().max()) == 0.0


def test_the_walk_still_takes_what_the_chunks_do_not():
    """Short steps, decays that are not worked out yet, keys of more than 128 entries and odd sizes: the same answers by the other kernel."""
    g, ops = torch.Generator(device="cuda"), Ops(torch.float32)
    g.manual_seed(1)
    for n, dk, ready in ((80, 64, True), (400, 64, False), (400, 132, True), (400, 62, True)):
        q, k, v = (torch.randn(n, d, generator=g, device="cuda") for d in (dk, dk, 16))
        z = torch.randn(n, dk, generator=g, device="cuda")
        decay = torch.sigmoid(z.double())
        want, _ = walk([n], 1, dk, 16, q.double()[:, None], k.double()[:, None], v.double()[:, None], decay[:, None])
        out, state = torch.full((n, 16), float("nan"), device="cuda"), torch.zeros(1, ops.recurrence_state_size("gated_linear", 1, dk, 16), device="cuda")
        ops.gated_recurrence("gated_linear", q, k, v, decay.float() if ready else z, out, state, starts([n]), i32([0]), 1, 1, 1, dk, 16, gates_ready=ready)
        assert rel(out, want[:, 0]) < 3e-6


@pytest.mark.parametrize("kind", ["retention", "retention finished", "matrix_memory", "delta_rule", "gated_linear"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("row,what", [(40, "v"), (43, "k"), (42, "kv"), (63, "v"), (1, "kv"), (97, "kv")])
def test_a_row_that_is_not_finite_reaches_no_row_before_it(kind, bad, row, what):
    """As in the row by row walk: the rows before it have the bits that they have beside finite rows, other heads and sequences too; the ones after it do not
    pass it off as finite."""
    g = torch.Generator(device="cuda")
    g.manual_seed(row)
    H, dk, dv, lens = 2, 64, 128, [130, 70]
    N = sum(lens)
    q, k, v, gate = (torch.randn(N, H * d, generator=g, device="cuda") for d in (dk, dk, dv, dv))
    memory = kind == "matrix_memory"
    gates = torch.randn(N, 2 * H, generator=g, device="cuda") + 3.0 if memory else torch.sigmoid(torch.randn(N, H * dk, generator=g, device="cuda") + 3.0)
    beta, decay = torch.sigmoid(torch.randn(N, H, generator=g, device="cuda")), torch.tensor([0.9, 0.97], device="cuda")
    if kind == "delta_rule":
        k = torch.nn.functional.normalize(k.view(N, H, dk), dim=-1).view(N, -1)
    ops = Ops(torch.float32)
    ops.CHUNK_MIN_ROWS = 1

    def run(k, v):
        out = torch.full((N, H * dv), float("nan"), device="cuda")
        if kind.startswith("retention"):
            state, done = torch.zeros(2, H, dk, dv, device="cuda"), kind.endswith("finished")
            ops.retention(q, k, v, out if done else None, state, starts(lens), i32(lens), i32([0, 1]), 2, decay, H, raw=torch.empty_like(out) if done else out,
                          raw_only=not done, **(dict(gate=gate, unit_norm_eps=1e-5) if done else {}))
        else:
            state = torch.zeros(2, ops.recurrence_state_size(kind, H, dk, dv), device="cuda")
            more = {"delta_rule": dict(beta=beta, a_log=torch.zeros(H, device="cuda"), dt_bias=torch.zeros(H * dk, device="cuda"), gates_ready=True),
                    "gated_linear": dict(gates_ready=True), "matrix_memory": dict(cap=15.0)}[kind]
            ops.gated_recurrence(kind, q, k, v, gates, out, state, starts(lens), i32([0, 1]), 2, H, H, dk, dv, **more)
        return out, state

    want, end = run(k, v)
    assert want.isfinite().all()
    k2, v2 = k.clone(), v.clone()
    if "k" in what:
        k2[row, 3] = bad
    if "v" in what:
        v2[row, 5] = bad
    got, end2 = run(k2, v2)
    assert torch.equal(got[:row], want[:row])                                           # the rows before, of both heads
    assert torch.equal(got[:, dv:], want[:, dv:]) and torch.equal(got[130:], want[130:]) and torch.equal(end2[1], end[1])       # the other head and sequence
    assert not got[row:130, 5].isfinite().any() and not end2[0].isfinite().all()


@pytest.mark.parametrize("kind", ["delta_rule", "gated_linear"])
@pytest.mark.parametrize("H,dk,dv,n", [(4, 128, 128, 700), (4, 64, 64, 300)])
def test_chunks_of_channel_decays_are_no_less_exact_than_the_walk(kind, H, dk, dv, n):
    """32-bit sums in another order: outputs within 15 % of the row by row kernel's error, states within 12 %, averaged over seeds."""
    g, delta = torch.Generator(device="cuda"), kind == "delta_rule"
    g.manual_seed(dk)
    sums = {True: [0.0, 0.0], False: [0.0, 0.0]}
    for _ in range(4):
        q, k, v = (torch.randn(n, H, d, generator=g, device="cuda") for d in (dk, dk, dv))
        z = torch.randn(n, H, dk, generator=g, device="cuda")
        if delta:
            k = torch.nn.functional.normalize(k, dim=-1)
            decay = torch.exp(-0.4 * torch.nn.functional.softplus(z - 1.0))
        else:
            decay = torch.sigmoid(z + 1.0) ** (1.0 / 12.0)
        beta = torch.sigmoid(torch.randn(n, H, generator=g, device="cuda"))
        want, (end,) = walk([n], H, dk, dv, q.double(), k.double(), v.double(), decay.double(), beta=beta.double() if delta else None)
        more = dict(beta=beta, a_log=torch.zeros(H, device="cuda"), dt_bias=torch.zeros(H * dk, device="cuda")) if delta else {}
        for chunks in (True, False):
            ops = Ops(torch.float32)
            ops.chunked_recurrences = chunks
            out, state = torch.empty(n, H * dv, device="cuda"), torch.zeros(1, ops.recurrence_state_size(kind, H, dk, dv), device="cuda")
            ops.gated_recurrence(kind, q.view(n, -1), k.view(n, -1), v.view(n, -1), decay.view(n, -1), out, state, starts([n]), i32([0]), 1, H, H, dk, dv,
                                 gates_ready=True, **more)
            sums[chunks][0] += rel(out.view(n, H, dv), want)
            sums[chunks][1] += rel(state[0][:H * dv * dk].view(H, dv, dk).transpose(1, 2), end)
    assert sums[True][0] < sums[False][0] * 1.15 and sums[True][1] < sums[False][1] * 1.12, sums


@pytest.mark.parametrize("kind", ["retention", "matrix_memory", "delta_rule", "gated_linear"])
def test_long_steps_go_in_spans_of_bounded_scratch(kind):
    """A list of chunks in spans gives the bits that it gives at once, whatever the spans cut; and scratch stays within its bound however long the step."""
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    H, dk, dv = 2, 64, 64
    memory = kind == "matrix_memory"

    def run(lens, budget=None):
        g.manual_seed(sum(lens))
        N, ops = sum(lens), Ops(torch.float32)
        ops.CHUNK_MIN_ROWS = 1
        if budget is not None:
            ops.CHUNK_WORK_BYTES = budget
        q, k, v = (torch.randn(N, H * d, generator=g, device="cuda") for d in (dk, dk, dv))
        gates = torch.randn(N, 2 * H, generator=g, device="cuda") + 3.0 if memory else torch.sigmoid(torch.randn(N, H * dk, generator=g, device="cuda") + 3.0)
        beta, decay = torch.sigmoid(torch.randn(N, H, generator=g, device="cuda")), torch.tensor([0.9, 0.97], device="cuda")
        if kind == "delta_rule":
            k = torch.nn.functional.normalize(k.view(N, H, dk), dim=-1).view(N, -1)
        out, st, sl, n = torch.full((N, H * dv), float("nan"), device="cuda"), starts(lens), i32(list(range(len(lens)))), len(lens)
        size = dk * dv * H if kind == "retention" else ops.recurrence_state_size(kind, H, dk, dv)
        state = torch.randn(n, size, generator=g, device="cuda") if not memory else torch.zeros(n, size, device="cuda")
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        if kind == "retention":
            ops.retention(q, k, v, None, state.view(n, H, dk, dv), st, i32(lens), sl, n, decay, H, raw=out, raw_only=True)
        else:
            more = {"delta_rule": dict(beta=beta, a_log=torch.zeros(H, device="cuda"), dt_bias=torch.zeros(H * dk, device="cuda"), gates_ready=True),
                    "gated_linear": dict(gates_ready=True), "matrix_memory": dict(cap=15.0)}[kind]
            ops.gated_recurrence(kind, q, k, v, gates, out, state, st, sl, n, H, H, dk, dv, **more)
        torch.cuda.synchronize()
        return out, state, torch.cuda.max_memory_allocated() - before

    whole, end, _ = run(LENS)
    per_place = H * (dk * dv + dk + 3) * 4 if memory else H * dk * dv * 4 if kind == "retention" else H * lib("chunked_channels").kvad_channels_work(dk, dv) * 4
    for places in (1, 2, 5):
        out, state, _ = run(LENS, places * per_place)
        assert torch.equal(out, whole) and torch.equal(state, end)
    budget = 16 * per_place
    out, state, peak = run([20000, 1, 300], budget)
    assert peak <= budget + (1 << 16), (peak, budget)
    assert out.isfinite().all()


@pytest.mark.parametrize("kind", ["retention", "retention finished", "matrix_memory", "delta_rule", "gated_linear"])
@pytest.mark.parametrize("dtype,dk,dv", [("float32", 64, 32), ("bfloat16", 128, 128)])
def test_short_sequences_keep_their_bits_beside_a_prompt(kind, dtype, dk, dv):
    """A prompt among decoding sequences goes in chunks, by the longest run; the sequences of fewer than 16 rows are walked and get what they get alone, to
    the bit, and so does the prompt."""
    if dtype == "bfloat16" and kind == "delta_rule":
        dtype = "float32"
    g = torch.Generator(device="cuda")
    g.manual_seed(dk)
    H, lens, t = 2, [1, 300, 1, 15, 16, 1], DT[dtype]
    N, ops, slots = sum(lens), Ops(t), [3, 0, 5, 1, 4, 2]
    q, k, v, gate = (torch.randn(N, H * d, generator=g, device="cuda").to(t) for d in (dk, dk, dv, dv))
    memory, done = kind == "matrix_memory", kind.endswith("finished")
    gates = torch.randn(N, 2 * H, generator=g, device="cuda") + 3.0 if memory else torch.sigmoid(torch.randn(N, H * dk, generator=g, device="cuda") + 3.0)
    beta, decay = torch.sigmoid(torch.randn(N, H, generator=g, device="cuda")), torch.tensor([0.9, 0.97], device="cuda")
    if kind == "delta_rule":
        k = torch.nn.functional.normalize(k.view(N, H, dk), dim=-1).view(N, -1)
    size = (H, dk, dv) if kind.startswith("retention") else (ops.recurrence_state_size(kind, H, dk, dv),)
    first = torch.randn(6, *size, generator=g, device="cuda") if not memory else torch.zeros(6, *size, device="cuda")
    at = [0] + list(np.cumsum(lens))

    def run(which, told):
        state, rows = first.clone(), torch.cat([torch.arange(at[i], at[i + 1], device="cuda") for i in which])
        pick, ls = (lambda x: x[rows].contiguous()), [lens[i] for i in which]
        raw, n = torch.full((len(rows), H * dv), float("nan"), device="cuda"), len(which)
        out = torch.full((len(rows), H * dv), float("nan"), device="cuda", dtype=t)
        more = dict(max_new=max(ls)) if told else {}
        if kind.startswith("retention"):
            ops.retention(pick(q), pick(k), pick(v), out if done else None, state, starts(ls), i32([x + 7 for x in ls]), i32([slots[i] for i in which]), n, decay, H,
                          raw=raw, raw_only=not done, **(dict(gate=pick(gate), unit_norm_eps=1e-5) if done else {}), **more)
        else:
            kw = {"delta_rule": dict(beta=pick(beta), a_log=torch.zeros(H, device="cuda"), dt_bias=torch.zeros(H * dk, device="cuda"), gates_ready=True),
                  "gated_linear": dict(gates_ready=True), "matrix_memory": dict(cap=15.0)}[kind]
            ops.gated_recurrence(kind, pick(q), pick(k), pick(v), pick(gates), raw, state, starts(ls), i32([slots[i] for i in which]), n, H, H, dk, dv, **kw, **more)
        return (out if done else raw), state

    got, state = run(range(6), True)
    assert got.isfinite().all()
    for i in range(6):
        alone, end = run([i], True)
        if i == 4:                                         # 16 rows: in chunks here, walked alone
            assert rel(got[at[4]:at[5]], alone.double()) < (5e-3 if done and dtype == "bfloat16" else 5e-5) and not torch.equal(state[slots[4]], end[slots[4]])
        else:
            assert torch.equal(got[at[i]:at[i + 1]], alone) and torch.equal(state[slots[i]], end[slots[i]]), i
    ops.chunked_recurrences = False
    walked, _ = run([1], True)
    assert not torch.equal(walked, got[at[1]:at[2]])       # (the prompt did go in chunks)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_gates_far_below_zero_of_chunked_retention(dtype):
    """silu(-88) is -5e-37: 1 + e^88 lies where a fast division gives 0."""
    g, ops = torch.Generator(device="cuda"), Ops(DT[dtype])
    g.manual_seed(3)
    q, k, v = (torch.randn(200, 2 * 64, generator=g, device="cuda").to(DT[dtype]) for _ in range(3))
    outs = []
    for z in (-88.0, 2.0):
        out, gate = (torch.full((200, 128), x, device="cuda", dtype=DT[dtype]) for x in (float("nan"), z))
        ops.retention(q, k, v, out, torch.zeros(1, 2, 64, 64, device="cuda"), i32([0, 200]), i32([200]), i32([0]), 1, torch.tensor([0.9, 1.0], device="cuda"), 2, gate=gate,
                      unit_norm_eps=1e-5, raw=torch.empty(200, 128, device="cuda"), max_new=200)
        outs.append(out.double() / (z * torch.sigmoid(torch.tensor(z, dtype=torch.float64))).item())
    assert rel(outs[0], outs[1]) < (6e-3 if dtype == "bfloat16" else 1e-6)      # (both rounded to the output's type; 32-bit exponentials and divisions)
