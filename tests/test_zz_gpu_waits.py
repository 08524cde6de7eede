"""Bounded waits of the tensor-core kernels that run out: reported by a counter, and harmless.  (In a file of its own that runs last: other tests ask that no wait has run out
in the process.)"""
import pytest
import torch

from kvad_b200.ops import Ops, linear_pieces_wait_timeouts, scored_prompt_wait_timeouts, scored_wide_wait_timeouts, wait_test_hooks
from tests.test_gpu_scored_wide import Case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,dtype,H,G,dk,dv", [("attention_scored_wide", torch.float32, 4, 2, 64, 64), ("attention_scored_wide", torch.float32, 2, 1, 128, 128),
                                                  ("attention_scored_prompt", torch.bfloat16, 4, 2, 64, 64), ("attention_scored_prompt", torch.bfloat16, 4, 1, 256, 256)])
def test_a_page_that_never_comes_is_reported_and_harmless(name, dtype, H, G, dk, dv):
    """The waits for it run out after the (shortened) limit, what is in flight is waited for, the launch returns without writing, and the next one is right."""
    count = scored_wide_wait_timeouts if dtype == torch.float32 else scored_prompt_wait_timeouts
    c, ops = Case([(200, 65), (70, 40)], H, G, dk, dv), Ops(dtype)
    c.q, c.kp, c.vp = (x.to(dtype) for x in (c.q.contiguous(), c.kp, c.vp))
    out = torch.full(c.out, 7.0, device="cuda")

    def run():
        ops.attention_scored(c.q, out, c.starts, c.lens, 2, c.max_new, c.table, c.kp, c.vp, H, c.scale)
        torch.cuda.synchronize()
    before = count()
    try:
        wait_test_hooks(name, 4096, True)
        run()
        assert count() > before and (out == 7.0).all()
    finally:
        wait_test_hooks(name)
    after = count()
    run()
    assert count() == after and out.isfinite().all()
    want = c.want()
    assert float((out.double() - want).norm() / want.norm()) < 1e-5


def test_weights_that_never_come_are_reported_and_harmless():
    """The waits for a block's weights run out after the (shortened) limit, copies in flight are waited for, the launch returns without writing, and the next one is right."""
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    ops = Ops(torch.float32)
    a, w = (torch.randn(*s, generator=g, device="cuda") for s in ((200, 512), (300, 512)))
    want = a.double() @ w.double().t()
    out = torch.full((200, 300), 7.0, device="cuda")
    before = linear_pieces_wait_timeouts()
    try:
        wait_test_hooks("linear_pieces", 4096, True)
        ops.linear(a, w, None, out)
        torch.cuda.synchronize()
        assert linear_pieces_wait_timeouts() > before and (out == 7.0).all()
    finally:
        wait_test_hooks("linear_pieces")
    after = linear_pieces_wait_timeouts()
    ops.linear(a, w, None, out)
    assert float((out.double() - want).norm() / want.norm()) < 1e-6 and linear_pieces_wait_timeouts() == after
