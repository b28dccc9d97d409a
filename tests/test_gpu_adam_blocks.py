"""The group update of csrc/optim.cu where its split into blocks can go wrong: sizes
about a block of 1,024 values, more blocks than a wave of CTAs takes at once, the
grid of four blocks a CTA (beyond 7.6 M values), a CTA that goes on to another parameter, and storage
that starts off a 16-byte boundary.  Compared with torch.optim.Adam: both hold the state in
FP32 and form the bias corrections in FP64, so one step of size lr = 0.01 differs by a few
roundings of the step (1e-2 x 1e-6) and half an ulp of the value (2.4e-7 up to 8): 1e-6 after two."""

import pytest
import torch

from diffsoup_b200.optimize import Adam

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize(
    "sizes", [(1,), (1023, 1024, 1025), (3, 760_001, 2, 5000), (2_000_003, 4096, 2_000_001), (5, 8_000_003, 1500)]
)
def test_update_equals_torch(sizes, shift):
    g = torch.Generator(device="cuda").manual_seed(len(sizes) + shift)
    room = [torch.randn(n + shift + 9, generator=g, device="cuda") for n in sizes]
    before = [r.clone() for r in room]
    ours = [r[shift : shift + n].requires_grad_() for r, n in zip(room, sizes)]
    theirs = [p.detach().clone().requires_grad_() for p in ours]
    oa, ob = Adam(ours, lr=1e-2), torch.optim.Adam(theirs, lr=1e-2)
    for _ in range(2):
        for p, q in zip(ours, theirs):
            q.grad = torch.randn(q.numel(), generator=g, device="cuda")
            p.grad = torch.cat([q.grad.new_zeros(shift), q.grad])[shift:]
        oa.step()
        ob.step()
    for p, q, r, b, n in zip(ours, theirs, room, before, sizes):
        torch.testing.assert_close(p, q, rtol=0, atol=1e-6)
        torch.testing.assert_close(oa.state[p]["exp_avg"], ob.state[q]["exp_avg"], rtol=1e-5, atol=1e-6)
        torch.testing.assert_close(oa.state[p]["exp_avg_sq"], ob.state[q]["exp_avg_sq"], rtol=1e-5, atol=1e-9)
        assert int(oa.state[p]["step"]) == 2
        assert torch.equal(r[:shift], b[:shift]) and torch.equal(r[shift + n :], b[shift + n :])
