"""The 32-bit latency form at the edges of its cluster sizes' ranges (4, 2 and 1 CTAs
per ciphertext) and the items form with two and three workers, for every digitG the
path takes, against the pipelines and the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int64)).cuda()


@pytest.fixture(scope="module", params=[(7, 4), (9, 3), (14, 2), (20, 2)])
def small(F, cuda_ok, request):
    from oracle_lib import Oracle
    P = F.params_preset(0)
    P.n, P.BG_bits, P.digitG = 7, request.param[0], request.param[1]
    F.derive(P)
    lsk, rsk = F.LWE_secretkey(P, 1), F.RLWE_secretkey(P, 2)
    bt, ks = F.bootstrap_key(P, 3, lsk, rsk), F.keyswitch_key(P, 4, rsk, lsk)
    with F.Context(P, 0) as ctx:
        ctx.upload_bootstrap_key(bt)
        ctx.upload_keyswitch_key(ks)
        yield P, ctx, lsk, bt, ks, Oracle.from_params(P)


@pytest.mark.parametrize("count", [1, 2, 35, 38, 39, 76, 77, 152, 153, 304, 380, 381, 1000])
def test_clusters(F, cuda_ok, small, count):
    torch = cuda_ok
    P, ctx, lsk, bt, ks, o = small
    rng = np.random.default_rng(count)
    ct = F.LWE_encrypt(P, 90 + count, lsk, rng.integers(0, 2, 2 * count, dtype=np.uint8))
    g = rng.integers(0, 6, count).astype(np.int32)
    d1, d2, dg = dev(torch, ct[:count]), dev(torch, ct[count:]), torch.from_numpy(g).cuda()
    for flags in (0, F.FLAG_FPGA_COMPAT, F.FLAG_FPGA_X1):
        got = []
        for solo in (-1, 0):
            ctx.set_option(F.OPT_BR_SOLO, solo)
            try:
                acc = torch.zeros((count, 2 * P.N), dtype=torch.int64, device="cuda")
                out = torch.zeros_like(d1)
                ctx.blind_rotate_async(d1.data_ptr(), d2.data_ptr(), dg.data_ptr(), count, acc.data_ptr(), flags)
                ctx.bootstrap_async(d1.data_ptr(), d2.data_ptr(), dg.data_ptr(), count, out.data_ptr(), flags)
                ctx.sync()
            finally:
                ctx.set_option(F.OPT_BR_SOLO, -1)
            got.append((acc, out))
        assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
        if flags == 0 and count <= 2:
            want, failed = o.eval_bootstrap_batch(ct[:count], ct[count:], g, bt, ks)
            assert failed == 0 and np.array_equal(got[0][1].cpu().numpy().view(np.uint64), want)


@pytest.mark.parametrize("bg,digits", [(7, 4), (9, 3), (14, 2)])
def test_items_of_a_gate(F, cuda_ok, bg, digits):
    """Gates of three items each (40 steps), at the edge of one worker per CTA, with two
    and with three: twice from the same scratch, against the pipelines."""
    torch = cuda_ok
    P = F.params_preset(0)
    P.n, P.BG_bits, P.digitG = 20, bg, digits
    F.derive(P)
    lsk, rsk = F.LWE_secretkey(P, 1), F.RLWE_secretkey(P, 2)
    with F.Context(P, 0) as ctx:
        ctx.upload_bootstrap_key(F.bootstrap_key(P, 3, lsk, rsk))
        ctx.upload_keyswitch_key(F.keyswitch_key(P, 4, rsk, lsk))
        for count in (200, 273, 274, 500):
            rng = np.random.default_rng(count)
            ct = F.LWE_encrypt(P, 7 + count, lsk, rng.integers(0, 2, 2 * count, dtype=np.uint8))
            d1, d2 = dev(torch, ct[:count]), dev(torch, ct[count:])
            dg = torch.from_numpy(rng.integers(0, 6, count).astype(np.int32)).cuda()
            for flags in (0, F.FLAG_FPGA_COMPAT, F.FLAG_FPGA_X1):
                got = []
                for solo in (-1, -1, 0):
                    ctx.set_option(F.OPT_BR_SOLO, solo)
                    acc = torch.zeros((count, 2 * P.N), dtype=torch.int64, device="cuda")
                    ctx.blind_rotate_async(d1.data_ptr(), d2.data_ptr(), dg.data_ptr(), count, acc.data_ptr(), flags)
                    ctx.sync()
                    got.append(acc)
                assert torch.equal(got[0], got[2]) and torch.equal(got[1], got[2]), (count, flags)
        assert ctx.device_status() == 0
