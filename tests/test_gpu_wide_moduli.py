"""The 64-bit path's two modular multiplications: Q = 2^b - c folds at 2^b
(b = 54 and the smallest b the rule takes with room for N = 2048's primes), any
other Q takes Shoup's form (just below and above the rule's range). Gadget
digits of 9 and of 27 bits. All words against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.uint64).view(np.int64)).cuda()


def host(t):
    return t.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("nbit,bg", [(47, 9), (50, 9), (53, 27), (54, 7), (54, 9), (54, 27), (55, 9), (57, 9)])
def test_moduli_vs_oracle(F, cuda_ok, nbit, bg):
    torch = cuda_ok
    from oracle_lib import Oracle
    P = F.params_preset(1)
    P.n, P.nbit, P.BG_bits = 3, nbit, bg
    P.Q = P.ROU = P.digitG = P.digitKS = P.digitKS_R = 0
    F.derive(P)
    o, Q = Oracle.from_params(P), int(P.Q)
    lsk, rsk = F.LWE_secretkey(P, 1), F.RLWE_secretkey(P, 2)
    bt, ks = F.bootstrap_key(P, 3, lsk, rsk), F.keyswitch_key(P, 4, rsk, lsk)
    rng = np.random.default_rng(nbit)
    with F.Context(P, 0) as ctx:
        ctx.upload_bootstrap_key(bt)
        assert ctx.verify_bootstrap_key(bt)
        ctx.upload_keyswitch_key(ks)
        # transforms, with edge words
        a = rng.integers(0, Q, (3, 2048), dtype=np.uint64)
        a[0] = Q - 1
        a[1, :4] = [0, 1, Q - 1, Q // 2]
        d = dev(torch, a)
        ctx.ntt_forward(d.data_ptr(), 3)
        torch.cuda.synchronize()
        assert np.array_equal(host(d), np.stack([o.ntt(x) for x in a]))
        ctx.ntt_inverse(d.data_ptr(), 3)
        torch.cuda.synchronize()
        assert np.array_equal(host(d), a)
        # products: split over the digits, and one CTA each with a shared RGSW
        for count in (2, 400):
            acc = rng.integers(0, Q, (count, 4096), dtype=np.uint64)
            acc[0] = Q - 1
            rgsw = rng.integers(0, Q, (1, P.digitG * 4 * 2048), dtype=np.uint64)
            rgsw[0, :4096] = Q - 1
            zero = dev(torch, np.zeros((count, 4096), dtype=np.uint64))
            da, dr, out = dev(torch, acc), dev(torch, rgsw), torch.zeros((count, 4096), dtype=torch.int64, device="cuda")
            # CMUX with c0 = 0 is the product itself
            ctx.CMUX(zero.data_ptr(), da.data_ptr(), dr.data_ptr(), out.data_ptr(), count)
            torch.cuda.synchronize()
            got = host(out)
            for i in (0, 1, count - 1):
                assert np.array_equal(got[i], o.rlwe_mult_rgsw(acc[i], rgsw[0])), (count, i)
        # automorphism and RLWE key switch
        c = acc[:2]
        ksk = rng.integers(0, Q, (int(P.digitKS_R), 2, 2048), dtype=np.uint64)
        dc, dk = dev(torch, c), dev(torch, ksk.reshape(-1))
        out = torch.zeros_like(dc)
        ctx.rlwe_substitute_async(dc.data_ptr(), 2, 3, out.data_ptr())
        ctx.sync()
        assert np.array_equal(host(out), np.stack([o.rlwe_substitute(x, 3) for x in c]))
        ctx.rlwe_keyswitch_async(dc.data_ptr(), 2, dk.data_ptr(), out.data_ptr())
        ctx.sync()
        assert np.array_equal(host(out), np.stack([o.rlwe_keyswitch(x, ksk) for x in c]))
        # whole gates, one CTA each and several per CTA
        bits = rng.integers(0, 2, 640, dtype=np.uint8)
        ct = F.LWE_encrypt(P, 5, lsk, bits)
        g = rng.integers(0, 6, 320).astype(np.int32)
        for count in (3, 320):
            c1, c2 = ct[:count], ct[320:320 + count]
            got = ctx.eval_bootstrap_batch(c1, c2, g[:count])
            want, failed = o.eval_bootstrap_batch(c1, c2, g[:count], bt, ks)
            assert failed == 0 and np.array_equal(got, want), count


@pytest.fixture(scope="module")
def small_wide(F, cuda_ok):
    P = F.params_preset(1)
    P.n = 5
    F.derive(P)
    lsk, rsk = F.LWE_secretkey(P, 1), F.RLWE_secretkey(P, 2)
    with F.Context(P, 0) as ctx:
        ctx.upload_bootstrap_key(F.bootstrap_key(P, 3, lsk, rsk))
        ctx.upload_keyswitch_key(F.keyswitch_key(P, 4, rsk, lsk))
        yield P, ctx, lsk


@pytest.mark.parametrize("count", [1, 8, 17, 18, 19, 38, 39, 76, 77, 152, 153, 305])
def test_forms_agree(F, cuda_ok, small_wide, count):
    """The latency form's cluster sizes at the edges of their ranges against the
    items form: accumulators and outputs, in the three issue orders."""
    torch = cuda_ok
    P, ctx, lsk = small_wide
    rng = np.random.default_rng(count)
    ct = F.LWE_encrypt(P, 40 + count, lsk, rng.integers(0, 2, 2 * count, dtype=np.uint8))
    d1, d2 = dev(torch, ct[:count]), dev(torch, ct[count:])
    dg = torch.from_numpy(rng.integers(0, 6, count).astype(np.int32)).cuda()
    for flags in (0, F.FLAG_FPGA_COMPAT, F.FLAG_FPGA_X1):
        got = []
        for pipes in (0, 2):
            ctx.set_option(F.OPT_BR_PIPES, pipes)
            try:
                acc = torch.zeros((count, 2 * P.N), dtype=torch.int64, device="cuda")
                out = torch.zeros_like(d1)
                ctx.blind_rotate_async(d1.data_ptr(), d2.data_ptr(), dg.data_ptr(), count, acc.data_ptr(), flags)
                ctx.bootstrap_async(d1.data_ptr(), d2.data_ptr(), dg.data_ptr(), count, out.data_ptr(), flags)
                ctx.sync()
            finally:
                ctx.set_option(F.OPT_BR_PIPES, 0)
            got.append((acc, out))
        assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.fixture(scope="module")
def longer_wide(F, cuda_ok):
    P = F.params_preset(1)
    P.n = 20   # 40 steps: three items of the latency form
    F.derive(P)
    lsk, rsk = F.LWE_secretkey(P, 1), F.RLWE_secretkey(P, 2)
    with F.Context(P, 0) as ctx:
        ctx.upload_bootstrap_key(F.bootstrap_key(P, 3, lsk, rsk))
        ctx.upload_keyswitch_key(F.keyswitch_key(P, 4, rsk, lsk))
        yield P, ctx, lsk


@pytest.mark.parametrize("count", [38, 39, 61, 64, 77, 100, 131, 134, 153, 200])
def test_cluster_items_agree(F, cuda_ok, longer_wide, count):
    """More gates than clusters that run at once: clusters that take items of the gates
    against the items form, in the three issue orders; twice, from the same scratch."""
    torch = cuda_ok
    P, ctx, lsk = longer_wide
    rng = np.random.default_rng(count)
    ct = F.LWE_encrypt(P, 70 + count, lsk, rng.integers(0, 2, 2 * count, dtype=np.uint8))
    d1, d2 = dev(torch, ct[:count]), dev(torch, ct[count:])
    dg = torch.from_numpy(rng.integers(0, 6, count).astype(np.int32)).cuda()
    for flags in (0, F.FLAG_FPGA_COMPAT, F.FLAG_FPGA_X1):
        got = []
        for pipes in (0, 0, 2):
            ctx.set_option(F.OPT_BR_PIPES, pipes)
            try:
                acc = torch.zeros((count, 2 * P.N), dtype=torch.int64, device="cuda")
                ctx.blind_rotate_async(d1.data_ptr(), d2.data_ptr(), dg.data_ptr(), count, acc.data_ptr(), flags)
                ctx.sync()
                got.append(host(acc))
            finally:
                ctx.set_option(F.OPT_BR_PIPES, 0)
        assert np.array_equal(got[0], got[2]) and np.array_equal(got[1], got[2]), flags
    assert ctx.device_status() == 0
