"""The split LWE key switch (each gate's rows over several CTAs, atomic partial sums)
against the one-CTA-per-gate and the tiled form, at both word widths: counts
around the split's slice rules."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[0, 1])
def small(F, cuda_ok, request):
    P = F.params_preset(request.param)
    P.n = 5
    F.derive(P)
    lsk, rsk = F.LWE_secretkey(P, 1), F.RLWE_secretkey(P, 2)
    with F.Context(P, 0) as ctx:
        ctx.upload_bootstrap_key(F.bootstrap_key(P, 3, lsk, rsk))
        ctx.upload_keyswitch_key(F.keyswitch_key(P, 4, rsk, lsk))
        yield P, ctx, lsk


@pytest.mark.parametrize("count", [1, 3, 151, 305, 607, 700])
def test_split_equals_other_forms(F, cuda_ok, small, count):
    torch = cuda_ok
    P, ctx, lsk = small
    rng = np.random.default_rng(count)
    ct = F.LWE_encrypt(P, 70 + count, lsk, rng.integers(0, 2, 2 * count, dtype=np.uint8))
    d = torch.from_numpy(ct.view(np.int64)).cuda()
    dg = torch.from_numpy(rng.integers(0, 6, count).astype(np.int32)).cuda()
    got = []
    for tiled in (-1, 0, 1):
        ctx.set_option(F.OPT_KS_TILED, tiled)
        try:
            out = torch.zeros((count, P.n + 1), dtype=torch.int64, device="cuda")
            ctx.bootstrap_async(d.data_ptr(), d[count:].data_ptr(), dg.data_ptr(), count, out.data_ptr())
            ctx.sync()
        finally:
            ctx.set_option(F.OPT_KS_TILED, -1)
        got.append(out)
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
