"""The autotuner against the launch shape that a context has by default."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPE = dict(regs_for_3=-1, ctas_per_sm=0, group=0, window=-1, pipes=0)


# Q of 55 bits: no fold form, the worker shapes with their window and groups
@pytest.mark.parametrize("preset,nbit,n,count", [(0, 27, 64, 1), (0, 27, 64, 300), (1, 54, 8, 1), (1, 54, 8, 100),
                                                 (1, 54, 8, 400), (1, 55, 8, 20)])
def test_default_is_tried(F, cuda_ok, preset, nbit, n, count):
    """The default shape is among the trials (the fastest trial is kept, or the default if
    that is within 1 %), no shape is tried twice, and the tuned context gives the words it gave before."""
    P = F.params_preset(preset)
    P.n, P.nbit = n, nbit
    P.Q = P.ROU = P.digitG = P.digitKS = P.digitKS_R = 0
    F.derive(P)
    lsk, rsk = F.LWE_secretkey(P, 1), F.RLWE_secretkey(P, 2)
    rng = np.random.default_rng(count)
    ct = F.LWE_encrypt(P, 6, lsk, rng.integers(0, 2, 2 * count, dtype=np.uint8))
    g = rng.integers(0, 6, count).astype(np.int32)
    with F.Context(P, 0) as ctx:
        ctx.upload_bootstrap_key(F.bootstrap_key(P, 3, lsk, rsk))
        ctx.upload_keyswitch_key(F.keyswitch_key(P, 4, rsk, lsk))
        before = ctx.eval_bootstrap_batch(ct[:count], ct[count:], g)
        trials = ctx.autotune(count)
        assert np.array_equal(ctx.eval_bootstrap_batch(ct[:count], ct[count:], g), before)
    shapes = [tuple(t[k] for k in SHAPE) for t in trials]
    assert shapes.count(tuple(SHAPE.values())) == 1, trials
    assert len(set(shapes)) == len(shapes) and all(t["ms"] > 0 for t in trials)
