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
