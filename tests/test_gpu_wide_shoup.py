"""The 64-bit blind rotation of the moduli without a fold form (Q of 55 and of 57
bits): one, two and three workers per CTA, several claim rounds, the remainder pool
and the step window on and off, the three issue orders, and a bounded wait that runs
out. All words against the oracle, or against the default launch of the same gates."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Keys:
    def __init__(self, F, nbit):
        from oracle_lib import Oracle
        P = F.params_preset(1)
        P.n, P.nbit = 6, nbit   # 12 steps
        P.Q = P.ROU = P.digitG = P.digitKS = P.digitKS_R = 0
        F.derive(P)
        self.F, self.P, self.oracle = F, P, Oracle.from_params(P)
        self.lsk, rsk = F.LWE_secretkey(P, 1), F.RLWE_secretkey(P, 2)
        self.bt, self.ks = F.bootstrap_key(P, 3, self.lsk, rsk), F.keyswitch_key(P, 4, rsk, self.lsk)

    def gates(self, count, seed):
        rng = np.random.default_rng(seed)
        ct = self.F.LWE_encrypt(self.P, 300 + seed, self.lsk, rng.integers(0, 2, 2 * count, dtype=np.uint8))
        return ct[:count], ct[count:], rng.integers(0, 6, count).astype(np.int32)

    def want(self, c1, c2, g, mode=0):
        out, _ = self.oracle.eval_bootstrap_batch(c1, c2, g, self.bt, self.ks, fpga_compat=mode)
        return out


@pytest.fixture(scope="module", params=[55, 57])
def shoup(F, cuda_ok, request):
    k = Keys(F, request.param)
    with F.Context(k.P, 0) as ctx:
        ctx.upload_bootstrap_key(k.bt)
        ctx.upload_keyswitch_key(k.ks)
        yield k, ctx


def options(F, ctx, pipes=0, window=-1, group=0, pool=-1):
    for o, v in ((F.OPT_BR_PIPES, pipes), (F.OPT_BR_WINDOW, window), (F.OPT_BR_GROUP, group), (F.OPT_BR_POOL, pool)):
        ctx.set_option(o, v)


def run(F, ctx, gates, flags=0, **shape):
    options(F, ctx, **shape)
    try:
        out = ctx.eval_bootstrap_batch(*gates, flags=flags)
        assert ctx.device_status() == 0
    finally:
        options(F, ctx)
    return out


@pytest.mark.parametrize("pipes,window", [(1, -1), (1, 0), (2, -1), (3, -1), (3, 0), (3, 4)])
def test_worker_shapes(F, shoup, pipes, window):
    """12 gates, and 13, which leave a remainder pool, in the three issue orders."""
    k, ctx = shoup
    for count in (12, 13):
        gates = k.gates(count, count)
        for flags, mode in ((0, 0), (F.FLAG_FPGA_COMPAT, 1), (F.FLAG_FPGA_X1, 2)):
            want = k.want(*gates, mode=mode)
            for pool in (-1, 0):
                got = run(F, ctx, gates, flags, pipes=pipes, window=window, pool=pool)
                assert np.array_equal(got, want), (count, flags, pool)


@pytest.mark.parametrize("pipes,group", [(0, 0), (1, 0), (2, 0), (3, 0), (3, 1), (2, 1)])
def test_batches(F, cuda_ok, shoup, pipes, group):
    """More gates than one per SM: a full grid with a pool, and 1000 gates, in several claim
    rounds with a group of one gate per worker."""
    k, ctx = shoup
    sms = cuda_ok.cuda.get_device_properties(0).multi_processor_count
    for count in (sms + 8, 2 * sms + 37, 1000):
        gates = k.gates(count, count)
        got = run(F, ctx, gates, pipes=pipes, group=group)
        assert np.array_equal(got, run(F, ctx, gates, pipes=pipes, group=group, pool=0)), count
        edges = [2 * sms - 1, 2 * sms] if count > 2 * sms else []   # the pool's side of the default launch
        idx = np.unique(np.append(np.linspace(0, count - 1, 12), edges).astype(int))
        assert np.array_equal(got[idx], k.want(*(x[idx] for x in gates))), count


def test_wait_expires(F, cuda_ok, shoup):
    """Two workers share a CTA's one gate: the second one's first wait runs out at a limit
    of zero polls, which the call reports; the context works again afterwards."""
    k, ctx = shoup
    gates = k.gates(1, 5)
    want = k.want(*gates)
    options(F, ctx, pipes=2)
    ctx.set_option(F.OPT_DEBUG_WAIT_LIMIT, 0)
    try:
        out, L = np.zeros_like(gates[0]), F.lib()
        p64 = ctypes.POINTER(ctypes.c_uint64)
        rc = L.fheacc_bootstrap(ctx.handle, gates[0].ctypes.data_as(p64), gates[1].ctypes.data_as(p64),
                                gates[2].ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), 1, out.ctypes.data_as(p64), 0)
        assert rc == F.EIO and b"bounded wait" in L.fheacc_last_error(ctx.handle)
    finally:
        ctx.set_option(F.OPT_DEBUG_WAIT_LIMIT, -1)
        options(F, ctx)
    assert np.array_equal(run(F, ctx, gates, pipes=2), want)


def test_rlwe_operations(F, cuda_ok, shoup):
    """expand_RLWE (its small levels split over transform pairs, the large ones not), the
    subs key's upload, and the RLWE blind rotation of few and of more RLWEs."""
    torch = cuda_ok
    k, ctx = shoup
    P, o, rng = k.P, k.oracle, np.random.default_rng(9)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.int64)).cuda()
    subs = rng.integers(0, P.Q, 11 * int(P.digitKS_R) * 2 * P.N, dtype=np.uint64)
    ctx.upload_subs_key(subs)
    assert ctx.verify_subs_key(subs) and ctx.verify_bootstrap_key(k.bt)
    c = rng.integers(0, P.Q, (60, 2 * P.N), dtype=np.uint64)
    rgsws = rng.integers(0, P.Q, 11 * P.digitG * 4 * P.N, dtype=np.uint64)
    dc, dr = dev(c), dev(rgsws)
    out = torch.zeros((P.N, 2 * P.N), dtype=torch.int64, device="cuda")
    ctx.expand_RLWE(dc.data_ptr(), out.data_ptr())
    ctx.sync()
    assert np.array_equal(out.cpu().numpy().view(np.uint64), o.expand_rlwe(c[0], subs))
    for count in (2, 60):
        for forward in (False, True):
            ctx.blind_rotate_RLWE(dc.data_ptr(), dr.data_ptr(), forward, out.data_ptr(), count)
            torch.cuda.synchronize()
            got = out[:count].cpu().numpy().view(np.uint64)
            for i in (0, count - 1):
                assert np.array_equal(got[i], o.rlwe_blind_rotate(c[i], forward, rgsws)), (count, forward)
