"""CMUX and RLWE x RGSW products whose outputs lie over inputs of other items: the
words of the same call with an output of its own."""
import pytest

pytestmark = pytest.mark.gpu


def uniform(torch, P, shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, P.Q, shape, dtype=torch.int64, device="cuda", generator=g)


@pytest.mark.parametrize("preset,count", [(0, 40), (1, 2), (1, 40), (1, 1000)])
def test_cmux_over_c1(F, cuda_ok, preset, count):
    """c1 of every other RLWE of an array, the outputs, contiguous, over its second half: an
    item's output is where a later item's c1 was."""
    torch = cuda_ok
    P = F.params_preset(preset)
    rw, gw = 2 * P.N, P.digitG * 4 * P.N
    c0, c1, sel = (uniform(torch, P, s, count + i) for i, s in enumerate([(2 * count, rw), (2 * count, rw), (gw,)]))
    with F.Context(P, 0) as ctx:
        want = torch.zeros((count, rw), dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        ctx.CMUX(c0.data_ptr(), c1.data_ptr(), sel.data_ptr(), want.data_ptr(), count, in_stride=2 * rw)
        torch.cuda.synchronize()
        over = c1[count:]
        ctx.CMUX(c0.data_ptr(), c1.data_ptr(), sel.data_ptr(), over.data_ptr(), count, in_stride=2 * rw)
        torch.cuda.synchronize()
        assert torch.equal(over, want)


@pytest.mark.parametrize("count", [2, 20])
def test_products_shifted(F, cuda_ok, count):
    """Outputs one RLWE further than the inputs (64-bit words)."""
    torch = cuda_ok
    P = F.params_preset(1)
    rw, gw = 2 * P.N, P.digitG * 4 * P.N
    acc, rgsw = uniform(torch, P, (count + 1, rw), count), uniform(torch, P, (count, gw), count + 1)
    with F.Context(P, 0) as ctx:
        want = torch.zeros((count, rw), dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        ctx.rlwe_mult_rgsw(acc.data_ptr(), rgsw.data_ptr(), want.data_ptr(), count)
        ctx.rlwe_mult_rgsw(acc.data_ptr(), rgsw.data_ptr(), acc[1:].data_ptr(), count)
        torch.cuda.synchronize()
        assert torch.equal(acc[1:], want)
