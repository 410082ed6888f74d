"""Bounded device waits of the blind rotations' latency and items forms that run out:
the key copies of a cluster, and a gate's items that wait for the item before.
FHEACC_OPT_DEBUG_WAIT_LIMIT shrinks the bounds: at zero polls every such wait expires;
at one to three a key copy may be seen in time by some threads of a CTA and not by
others, which decide as one. The kernel always returns, with the right words or with
FHEACC_STATUS_WAIT_LIMIT, and the context works again once the limit is restored.
Nothing here faults or hangs a GPU: the waits end by their own bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(F, preset, n):
    P = F.params_preset(preset)
    P.n = n
    F.derive(P)
    lsk, rsk = F.LWE_secretkey(P, 1), F.RLWE_secretkey(P, 2)
    ctx = F.Context(P, 0)
    ctx.upload_bootstrap_key(F.bootstrap_key(P, 3, lsk, rsk))
    ctx.upload_keyswitch_key(F.keyswitch_key(P, 4, rsk, lsk))
    return P, ctx, lsk


@pytest.fixture(scope="module")
def wide(F, cuda_ok):
    P, ctx, lsk = make(F, 1, 20)   # 40 steps: three items of a gate
    yield P, ctx, lsk
    ctx.close()


def expire(F, torch, P, ctx, lsk, count, limit, must):
    """The gates with the limit and, before and after, without it."""
    L = F.lib()
    rng = np.random.default_rng(count)
    ct = F.LWE_encrypt(P, 20 + count, lsk, rng.integers(0, 2, 2 * count, dtype=np.uint8))
    d = torch.from_numpy(ct.view(np.int64)).cuda()
    dg = torch.from_numpy(rng.integers(0, 6, count).astype(np.int32)).cuda()
    out = torch.zeros((count, P.n + 1), dtype=torch.int64, device="cuda")

    def run():
        out.zero_()
        torch.cuda.synchronize()
        ctx.bootstrap_async(d.data_ptr(), d[count:].data_ptr(), dg.data_ptr(), count, out.data_ptr())
        return L.fheacc_sync(ctx.handle, 60000)

    assert run() == F.OK
    want = out.clone()
    ctx.set_option(F.OPT_DEBUG_WAIT_LIMIT, limit)
    try:
        for _ in range(3):
            rc = run()
            assert rc == F.EIO if must else rc in (F.OK, F.EIO)
            if rc == F.OK:
                assert torch.equal(out, want)
            else:
                assert b"bounded wait" in L.fheacc_last_error(ctx.handle)
    finally:
        ctx.set_option(F.OPT_DEBUG_WAIT_LIMIT, -1)
    assert run() == F.OK and torch.equal(out, want)


@pytest.mark.parametrize("count", [1, 30, 70, 100, 200])
@pytest.mark.parametrize("limit", [0, 1, 2, 3])
def test_wide_clusters(F, cuda_ok, wide, count, limit):
    """8, 4 and 2 CTAs a gate, and items of more gates than clusters that run at once."""
    expire(F, cuda_ok, *wide, count, limit, limit == 0)


@pytest.fixture(scope="module")
def narrow(F, cuda_ok):
    P, ctx, lsk = make(F, 0, 20)   # 40 steps: three or five items of a gate
    yield P, ctx, lsk
    ctx.close()


@pytest.mark.parametrize("limit", [0, 1, 2, 3])
def test_narrow_items(F, cuda_ok, narrow, limit):
    """One worker per CTA (whole keys copied), two (no copies; more workers than gates, so
    the surplus ones wait for a gate's item before) and three (a part of the keys)."""
    sms = cuda_ok.cuda.get_device_properties(0).multi_processor_count
    narrow[1].set_option(F.OPT_BR_SOLO, 1)   # the items form, also with a limit
    try:
        for count in (sms + 8, 2 * sms - 20, 3 * sms):
            expire(F, cuda_ok, *narrow, count, limit, limit == 0)
    finally:
        narrow[1].set_option(F.OPT_BR_SOLO, -1)
