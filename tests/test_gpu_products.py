"""Fused CMUX / RLWE x RGSW products of the 64-bit path at the edges of their forms'
ranges (clusters of 8, 4, 2 CTAs, one CTA, workers), one RGSW for all or one each,
output over an input: against the oracle and against one-product calls."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def wide(F, cuda_ok):
    from oracle_lib import Oracle
    P = F.params_preset(1)
    with F.Context(P, 0) as ctx:
        yield P, ctx, Oracle.from_params(P)


@pytest.mark.parametrize("count", [1, 8, 19, 20, 38, 39, 76, 77, 152, 153, 310])
def test_cmux_forms(F, cuda_ok, wide, count):
    torch = cuda_ok
    P, ctx, o = wide
    rw, gw = 2 * P.N, P.digitG * 4 * P.N
    g = torch.Generator(device="cuda").manual_seed(count)
    v = torch.randint(0, P.Q, (2 * count, rw), dtype=torch.int64, device="cuda", generator=g)
    v[0] = P.Q - 1
    v[1] = 0
    each = count <= 39
    sel = torch.randint(0, P.Q, (count if each else 1, gw), dtype=torch.int64, device="cuda", generator=g)
    out = torch.zeros((count, rw), dtype=torch.int64, device="cuda")
    ctx.CMUX(v.data_ptr(), v.data_ptr() + 8 * rw, sel.data_ptr(), out.data_ptr(), count, in_stride=2 * rw,
             sel_shared=not each)
    # contiguous inputs, output over c0, and over c1
    c0, c1 = v[0::2].contiguous(), v[1::2].contiguous()
    d0, d1 = c0.clone(), c1.clone()
    ctx.CMUX(d0.data_ptr(), c1.data_ptr(), sel.data_ptr(), d0.data_ptr(), count, sel_shared=not each)
    ctx.CMUX(c0.data_ptr(), d1.data_ptr(), sel.data_ptr(), d1.data_ptr(), count, sel_shared=not each)
    torch.cuda.synchronize()
    assert torch.equal(d0, out) and torch.equal(d1, out)
    for k in sorted({0, count // 2, count - 1}):
        s = sel[k if each else 0]
        one = torch.zeros(rw, dtype=torch.int64, device="cuda")
        ctx.CMUX(c0[k].data_ptr(), c1[k].data_ptr(), s.data_ptr(), one.data_ptr(), 1)
        torch.cuda.synchronize()
        assert torch.equal(one, out[k])
    host = [x.cpu().numpy().view(np.uint64) for x in (v[0], v[1], sel[0], out[0])]
    assert np.array_equal(o.cmux(host[0], host[1], host[2]), host[3])
