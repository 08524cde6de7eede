"""Experts' products of few rows: the block's weights by one bulk copy, bfloat16 on the tensor cores."""
import pytest
import torch

from kvad_b200.ops import Ops, lib

pytestmark = pytest.mark.gpu
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}


# K that ends inside a warp's 32 and inside the block's 256, one piece of K, outputs that end inside a block of 16, K whose rows fit a block
# sixteen, eight, four at a time and not at all
@pytest.mark.parametrize("dtype,n_out,k", [("bfloat16", 16, 256), ("bfloat16", 17, 8), ("bfloat16", 33, 264), ("bfloat16", 5, 1408), ("bfloat16", 40, 6400),
                                           ("bfloat16", 20, 6408), ("bfloat16", 9, 13000), ("float32", 17, 4), ("float32", 40, 260), ("float32", 33, 1408),
                                           ("float32", 20, 6404), ("float32", 9, 13000), ("float32", 7, 51204)])
@pytest.mark.parametrize("lists", [False, True])
def test_few_rows_of_experts_are_no_further_off_than_the_fmaf_chain(dtype, n_out, k, lists):
    g = torch.Generator(device="cuda")
    g.manual_seed(n_out * k)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    ops, h = Ops(DT[dtype]), lib("moe")
    TM, used = h.kvad_moe_tile_rows(), [1, 2, 4, 8, 9, 32, 0, 3]
    tiles = len(used)
    experts = [2, 0, 1, 1, 2, 0, 1, -1]                      # (the last tile belongs to nobody; one has no rows)
    valid = torch.full((tiles, TM), -1, dtype=torch.int32)
    for t, n in enumerate(used):
        valid[t, torch.randperm(TM, generator=torch.Generator().manual_seed(t))[:n]] = 1
    P = tiles * TM
    a = rnd(P + 3, k + 8).to(DT[dtype])[:, :k]
    w = (rnd(3, n_out, k) * 0.3).to(DT[dtype])
    to = torch.randperm(P, generator=torch.Generator().manual_seed(1)).int().cuda() if lists else None
    frm = torch.randint(0, P + 3, (P,), generator=torch.Generator().manual_seed(2)).int().cuda() if lists else None
    if not lists:
        a = a[:P]
    flat = valid.flatten().cuda()
    live = [p for p in range(P) if flat[p] >= 0 and experts[p // TM] >= 0]
    src = [int(frm[p]) if lists else p for p in live]
    dst = [int(to[p]) if lists else p for p in live]
    want = torch.stack([w[experts[p // TM]].double() @ a[s].double() for p, s in zip(live, src)])
    te, size = torch.tensor(experts, dtype=torch.int32, device="cuda"), torch.stack([w[experts[p // TM]].double().abs() @ a[s].double().abs() for p, s in zip(live, src)])
    for out_dtype in {DT[dtype], torch.float32}:
        got = []
        for few in (True, False):
            out = torch.full((P, n_out), float("nan"), dtype=out_dtype, device="cuda")
            ops.grouped_linear(a, w, out, te, flat, in_rows=frm, out_rows=to, few_rows=few)
            rest = torch.ones(P, dtype=torch.bool)
            rest[dst] = False
            assert out[rest.cuda()].isnan().all()             # nobody else's rows are written
            got.append(out[dst].double())
        # sums of k products in 32 bits: 16 roundings deep where lanes and warps share them, k / 256 + 16 at most; and the output's own rounding
        bound = size * (k / 256 + 16) * 2.0 ** -23 + want.abs() * (2.0 ** -8 if out_dtype == torch.bfloat16 else 0)
        assert ((got[0] - want).abs() <= bound).all()
        few, chain = ((x - want).norm() / want.norm() for x in got)
        assert few <= 1.05 * chain + 2.0 ** -25               # (both are sums of rounding errors of a few hundred outputs)
    assert h.kvad_moe_status() == 0


@pytest.mark.parametrize("dtype,k", [("bfloat16", 256), ("bfloat16", 6408), ("float32", 256), ("float32", 13000)])
def test_a_copy_that_never_comes_is_reported_and_writes_nothing(dtype, k):
    """The bounded wait for a block's weights, on the tensor cores and off: with the copies left out it gives up by counting, the counter rises and no output
    is written; the launch after it is ordinary.  (The 32-bit product's counter has its reader too.)"""
    from kvad_b200.ops import linear_split_wait_timeouts, moe_test_hooks, moe_wait_timeouts
    g = torch.Generator(device="cuda")
    g.manual_seed(k)
    ops, TM, n_out = Ops(DT[dtype]), lib("moe").kvad_moe_tile_rows(), 20
    a, w = torch.randn(TM, k, generator=g, device="cuda").to(DT[dtype]), torch.randn(1, n_out, k, generator=g, device="cuda").to(DT[dtype])
    te, flat = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.full((TM,), -1, dtype=torch.int32, device="cuda")
    flat[:11] = 1
    out = torch.full((TM, n_out), 7.0, dtype=DT[dtype], device="cuda")
    before, split = moe_wait_timeouts(), linear_split_wait_timeouts()
    try:
        moe_test_hooks(wait_limit=200, skip_copies=True)
        ops.grouped_linear(a, w, out, te, flat, few_rows=True)
        torch.cuda.synchronize()
        assert moe_wait_timeouts() > before and bool((out == 7.0).all())
    finally:
        moe_test_hooks()
    again = moe_wait_timeouts()
    ops.grouped_linear(a, w, out, te, flat, few_rows=True)
    want = a[:11].double() @ w[0].double().t()
    assert ((out[:11].double() - want).norm() / want.norm()).item() < (5e-3 if dtype == "bfloat16" else 1e-6) and bool((out[11:] == 7.0).all())
    assert moe_wait_timeouts() == again and linear_split_wait_timeouts() == split
