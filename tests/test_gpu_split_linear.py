"""The 32-bit product on the tensor cores (operands cut into bfloat16 pieces) and the head-wise maps of many rows in one launch."""
import pytest
import torch

from kvad_b200.ops import Ops, lib

pytestmark = pytest.mark.gpu
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}


def rel(got, ref):
    return float((got.double() - ref).norm() / ref.norm())


def randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda")


# edges of tiles (128 rows, 64 or 128 outputs), of a block of K (32) and of the four slots, the shortest K, one row past a tile,
# more tiles than SMs (a CTA goes round its slots over several tiles)
@pytest.mark.parametrize("m,n,k", [(33, 64, 4), (64, 65, 32), (127, 128, 36), (128, 200, 128), (129, 63, 160), (300, 1031, 96), (1500, 2309, 200), (70, 5, 772)])
@pytest.mark.parametrize("tile", [64, 128])
@pytest.mark.parametrize("pieces", [False, True])
def test_split_product_is_no_further_off_than_the_fmaf_chain(m, n, k, tile, pieces):
    """Either road by itself: weights cut where they are used (linear_split), or by a pass before (linear_pieces)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(m * n + k)
    ops, chain = Ops(torch.float32), Ops(torch.float32)
    chain.split_linear, chain.rows_linear_max, ops.SPLIT_MIN_ROWS = False, 0, 1
    ops.pieces_linear, ops.PIECES_MIN_ROWS, ops.PIECES_MIN_K = pieces, 1, 1
    wide = randn(g, m, k + 8)
    a, w, b, old = wide[:, 4:4 + k], randn(g, n, k) * 0.3, randn(g, n), randn(g, m, n + 3)[:, :n]
    exact = a.double() @ w.double().t()
    for epi in ("store", "gelu_tanh", "gelu_erf", "residual", "store_f32"):
        want = exact + b.double()
        if epi.startswith("gelu"):
            want = torch.nn.functional.gelu(want, approximate="tanh" if epi == "gelu_tanh" else "none")
        if epi == "residual":
            want = want + old.double()
        outs = []
        for o, t in ((ops, tile), (chain, 0)):
            out = torch.full((m, n + 3), float("nan"), device="cuda")
            out[:, :n] = old
            o.linear(a, w, b, out[:, :n], epi, tile=t)
            assert torch.isnan(out[:, n:]).all()
            outs.append(rel(out[:, :n], want))
        # six products leave out less than 2^-23 of |a||w|; single roundings of the result are 2^-25 on average
        assert outs[0] < max(1.1 * outs[1], 1.5e-7), (epi, outs)
    assert lib("linear_split").kvad_linear_split_status() == 0 and lib("linear_pieces").kvad_linear_pieces_status() == 0


def test_split_product_of_values_that_bfloat16_cannot_hold():
    """Pieces down to the last bit; infinities, NaN and overflow as the fmaf chain gives them; a row's bits whatever its company."""
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    ops, chain = Ops(torch.float32), Ops(torch.float32)
    chain.split_linear = False
    a, w = torch.ones(200, 64, device="cuda"), torch.zeros(96, 64, device="cuda")
    a[:, 0] = 1.0 + 2.0 ** -23 * torch.arange(1, 201, device="cuda")
    w[:, 0] = 1.0
    out = torch.empty(200, 96, device="cuda")
    ops.linear(a, w, None, out)
    assert torch.equal(out, a[:, :1].expand(200, 96))                     # a product with 1.0 is exact
    a, w = randn(g, 200, 64), randn(g, 96, 64)
    a[3, 5], a[7, 1], a[11, 0], a[20, 0], w[30, 0], w[9, 5], w[9, 0] = float("inf"), float("nan"), -float("inf"), 3e38, 3e38, 0.0, 1.0
    got, want = torch.empty(200, 96, device="cuda"), torch.empty(200, 96, device="cuda")
    ops.linear(a, w, None, got)
    chain.linear(a, w, None, want)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    fine = torch.isfinite(want)
    assert bool((got[~fine & ~torch.isnan(want)] == want[~fine & ~torch.isnan(want)]).all()) and rel(got[fine][None], want[fine][None].double()) < 1e-6
    few = torch.empty(70, 96, device="cuda")
    ops.linear(a[100:170], w, None, few)
    assert torch.equal(few, got[100:170])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("n,H,n_in,n_out,pad", [(65, 3, 64, 256, 0), (129, 16, 32, 64, 16), (300, 2, 72, 40, 8), (1030, 5, 136, 200, 24), (70, 1, 8, 300, 0), (130, 3, 12, 20, 4)])
def test_head_maps_of_many_rows_in_one_launch(dtype, n, H, n_in, n_out, pad):
    g = torch.Generator(device="cuda")
    g.manual_seed(n + n_in)
    ops, t = Ops(DT[dtype]), DT[dtype]
    a, w = randn(g, n, H * (n_in + pad)).to(t), (randn(g, H, n_out, n_in) * n_in ** -0.5).to(t)
    a.view(n, H, -1)[:, :, n_in:] = float("nan")                          # what lies between the heads is nobody's
    out = torch.full((n, H * (n_out + pad) + 8), float("nan"), device="cuda", dtype=t)
    ops.linear_heads(a, w, out, head_stride_a=n_in + pad, head_stride_out=n_out + pad)
    got = out[:, :H * (n_out + pad)].view(n, H, -1)
    want = torch.einsum("rhi,hji->rhj", a.view(n, H, -1)[:, :, :n_in].double(), w.double())
    assert rel(got[:, :, :n_out], want) < (2e-7 if dtype == "float32" else 3e-3)      # bfloat16: one rounding, 2^-9 at most
    assert torch.isnan(got[:, :, n_out:]).all() and torch.isnan(out[:, H * (n_out + pad):]).all()
    gate = randn(g, n, H * n_out).to(t)
    gated = torch.empty(n, H * n_out, device="cuda", dtype=t)
    ops.linear_heads(a, w, gated, head_stride_a=n_in + pad, head_stride_out=n_out, gate=gate)
    assert rel(gated.view(n, H, n_out), want * torch.sigmoid(gate.double()).view(n, H, n_out)) < (3e-7 if dtype == "float32" else 5e-3)


@pytest.mark.parametrize("tile", [16, 32, 96, 192, 256])
def test_a_tile_width_of_the_other_kernels_is_the_split_products_own_choice(tile):
    """`tile` fixes the width of the bfloat16 kernel's tiles; the 32-bit product has 64 and 128 only and takes no notice of others."""
    g = torch.Generator(device="cuda")
    g.manual_seed(tile)
    ops, a, w = Ops(torch.float32), randn(g, 200, 64), randn(g, 300, 64)
    want, got = torch.empty(200, 300, device="cuda"), torch.empty(200, 300, device="cuda")
    ops.linear(a, w, None, want)
    ops.linear(a, w, None, got, tile=tile)
    assert torch.equal(got, want)


# one row past a tile, ends of tiles of every width, K that ends within a block of 32 and within an odd one, more tiles than SMs (a CTA's rings run on)
@pytest.mark.parametrize("m,n,k", [(65, 1, 256), (128, 193, 260), (129, 64, 300), (257, 385, 512), (1500, 2309, 292), (70, 130, 772)])
@pytest.mark.parametrize("tile", [64, 128, 192])
def test_product_of_cut_weights_has_the_split_products_bits(m, n, k, tile):
    from kvad_b200.ops import linear_pieces_wait_timeouts
    g = torch.Generator(device="cuda")
    g.manual_seed(m + n * k)
    ops, split = Ops(torch.float32), Ops(torch.float32)
    split.pieces_linear, ops.PIECES_MIN_K = False, 1
    a, w, b, old = randn(g, m, k + 8)[:, 4:4 + k], randn(g, n, k) * 0.3, randn(g, n), randn(g, m, n + 3)[:, :n]
    strange = a.clone()
    strange[m // 2, 3], strange[m - 1, k - 1] = float("inf"), float("nan")
    for x, epi in ((a, "store"), (a, "gelu_tanh"), (a, "gelu_erf"), (a, "residual"), (strange, "store")):
        outs = []
        for o, t in ((ops, tile), (split, 0)):
            out = torch.full((m, n + 3), float("nan"), device="cuda")
            out[:, :n] = old
            o.linear(x, w, b, out[:, :n], epi, tile=t)
            assert torch.isnan(out[:, n:]).all()
            outs.append(out[:, :n].clone())
        assert torch.equal(outs[0].nan_to_num(7.0), outs[1].nan_to_num(7.0)) and torch.equal(outs[0].isnan(), outs[1].isnan())
    assert linear_pieces_wait_timeouts() == 0


def roads(monkeypatch, call):
    """Which of the two libraries the products of `call` went to."""
    import kvad_b200.ops as module
    seen, real = [], module.lib
    monkeypatch.setattr(module, "lib", lambda name: (seen.append(name), real(name))[1])
    call()
    return [x for x in seen if x in ("linear_split", "linear_pieces")]


@pytest.mark.parametrize("m,n,k,road", [(65, 4804, 256, "split"), (128, 4800, 256, "pieces"), (128, 4096, 2052, "split"), (128, 3072, 4096, "pieces"), (129, 4804, 256, "pieces"),
                                        (64, 300, 256, ""), (70, 300, 252, "split")])
def test_which_road_a_product_takes(monkeypatch, m, n, k, road):
    """One tile of rows and many outputs: the weights are cut where they are used; either way the same bits."""
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    ops, split = Ops(torch.float32), Ops(torch.float32)
    split.pieces_linear = False
    a, w = randn(g, m, k), randn(g, n, k)
    outs = [torch.full((m, n), float("nan"), device="cuda") for _ in range(2)]
    assert roads(monkeypatch, lambda: ops.linear(a, w, None, outs[0])) == (["linear_" + road] if road else [])
    split.linear(a, w, None, outs[1])
    assert torch.equal(*outs) and outs[0].isfinite().all()


def test_a_product_without_room_for_its_scratch_runs_all_the_same(monkeypatch):
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    ops = Ops(torch.float32)
    a, w, real = randn(g, 200, 512), randn(g, 700, 512), torch.empty
    want, got = (torch.full((200, 700), float("nan"), device="cuda") for _ in range(2))
    assert roads(monkeypatch, lambda: ops.linear(a, w, None, want)) == ["linear_pieces"]

    def none_left(*args, **kw):
        if kw.get("dtype") == torch.uint8:
            raise torch.cuda.OutOfMemoryError("no room")
        return real(*args, **kw)
    monkeypatch.setattr(torch, "empty", none_left)
    assert roads(monkeypatch, lambda: ops.linear(a, w, None, got)) == ["linear_split"]
    assert torch.equal(got, want)
    ops.PIECES_WORK_BYTES = 1 << 16
    monkeypatch.setattr(torch, "empty", real)
    assert roads(monkeypatch, lambda: ops.linear(a, w, None, got)) == ["linear_split"]
