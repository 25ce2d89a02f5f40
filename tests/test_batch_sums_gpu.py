"""Sums over a short batch: volumes and batches at the edges of both CTA shapes, against fp64."""
import pytest
import torch

import primitiv_b200 as pb

pytestmark = pytest.mark.gpu

# one CTA, ragged and whole tiles, the most that takes the many-lane form and the first beyond it
VOLUMES = [1, 7, 10, 33, 128, 132, 800, 2368, 9472, 9476]
BATCHES = [63, 64, 65, 200, 255, 256]


@pytest.mark.parametrize("half", [False, True], ids=["fp32", "fp16"])
@pytest.mark.parametrize("offset", [0, 1], ids=["aligned", "unaligned"])
def test_gradient_of_a_broadcast_operand_and_batch_sum(ctx, half, offset):
    mode, kind = (pb.MODE_FP16, torch.float16) if half else (pb.MODE_FP32_3XTF32, torch.float32)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(2)
    make = lambda n: torch.randn(n + 9, device="cuda", generator=gen).to(kind)[offset:]
    # sums in fp32 of up to 256 terms, rounded once to the storage type
    bound = lambda terms, want: terms.abs().sum(0) * 256 * 2.0 ** -24 + want.abs() * 2.0 ** (-11 if half else -24) + (6e-8 if half else 0)
    for volume in VOLUMES:
        for batch in BATCHES:
            n = volume * batch
            for op in (0, 2):                      # add, multiply
                for summed in (0, 1):               # which operand has no batch
                    sizes = (volume, n) if summed == 0 else (n, volume)
                    a, b, gy, y = make(sizes[0]), make(sizes[1]), make(n), make(n)
                    ga, gb = make(sizes[0]), make(sizes[1])
                    old = (ga, gb)[summed].double()
                    ctx.op("b200_binary_bw", mode, op, a.data_ptr(), b.data_ptr(), y.data_ptr(), gy.data_ptr(), ga.data_ptr(), gb.data_ptr(),
                           volume, batch, summed, 1 - summed, 1, 1, None)
                    other = (b, a)[summed].double()[:n].view(batch, volume) if op == 2 else 1.0
                    terms = gy.double()[:n].view(batch, volume) * other
                    got, want = (ga, gb)[summed].double(), old[:volume] + terms.sum(0)
                    assert ((got[:volume] - want).abs() <= bound(terms, want)).all(), (volume, batch, op, summed)
                    assert torch.equal(got[volume:], old[volume:]), "wrote past the gradient"
            x, s = make(n), make(volume)
            after = s[volume:].clone()
            ctx.op("b200_batch_sum_fw", mode, x.data_ptr(), s.data_ptr(), volume, batch, None)
            terms = x.double()[:n].view(batch, volume)
            assert ((s.double()[:volume] - terms.sum(0)).abs() <= bound(terms, terms.sum(0))).all(), (volume, batch)
            assert torch.equal(s[volume:], after)
    assert ctx.status_poll() == 0
