"""Refresh bases whose residues do not fit a byte are refused with their key (a gate
would take a wrong row of it); all others give the oracle's words."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def params(F, preset, q, Br):
    P = F.params_preset(preset)
    P.n, P.q, P.Br, P.digitR = 2, q, Br, 0
    for i in range(6):
        P.gate_constant[i] = 0
    P.E = 0
    F.derive(P)
    return P


@pytest.mark.parametrize("preset", [0, 1])
def test_residues_of_a_byte(F, cuda_ok, preset):
    from oracle_lib import Oracle
    for q, Br, ok in ((512, 256, True), (256, 300, True), (512, 257, False), (512, 512, False)):
        P = params(F, preset, q, Br)
        lsk, rsk = F.LWE_secretkey(P, 1), F.RLWE_secretkey(P, 2)
        bt, ks = F.bootstrap_key(P, 3, lsk, rsk), F.keyswitch_key(P, 4, rsk, lsk)
        with F.Context(P, 0) as ctx:
            if not ok:
                with pytest.raises(F.FheaccError, match="refresh base"):
                    ctx.upload_bootstrap_key(bt)
                continue
            ctx.upload_bootstrap_key(bt)
            ctx.upload_keyswitch_key(ks)
            rng = np.random.default_rng(q + Br)
            for count in (3, 200):
                ct = F.LWE_encrypt(P, count, lsk, rng.integers(0, 2, 2 * count, dtype=np.uint8))
                g = rng.integers(0, 6, count).astype(np.int32)
                got = ctx.eval_bootstrap_batch(ct[:count], ct[count:], g)
                want, _ = Oracle.from_params(P).eval_bootstrap_batch(ct[:count], ct[count:], g, bt, ks)
                assert np.array_equal(got, want), (q, Br, count)
