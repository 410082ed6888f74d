"""The LWE key switch at bases whose digits take one byte (up to 256), two (up to
65536) and four, at both word widths: the kernel of one CTA per ciphertext (the
key-switch call) and the split kernel (batches of gates), word for word against
the oracle. The tiled kernels take bases up to 255 only."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int64)).cuda()


# (preset, base, digits: 0 as many as Q needs); a base above 65536 with one digit, to keep the key at 1 GB
@pytest.mark.parametrize("preset,base,digits", [(0, 2, 0), (0, 256, 0), (0, 257, 0), (0, 512, 0), (0, 1000, 0),
                                                (0, 65537, 1), (1, 256, 0), (1, 257, 0), (1, 512, 0)])
def test_bases(F, cuda_ok, preset, base, digits):
    from oracle_lib import Oracle
    torch = cuda_ok
    P = F.params_preset(preset)
    P.n, P.Bks, P.digitKS = (1 if base > 65536 else 5), base, digits
    F.derive(P)
    o, rng = Oracle.from_params(P), np.random.default_rng(base)
    lsk, rsk = F.LWE_secretkey(P, 1), F.RLWE_secretkey(P, 2)
    bt = F.bootstrap_key(P, 3, lsk, rsk)
    # the key switch is a sum of the rows that the digits select, whatever the rows hold
    ks = rng.integers(0, P.Q, base * P.digitKS * P.N * (P.n + 1), dtype=np.uint64)
    with F.Context(P, 0) as ctx:
        ctx.upload_bootstrap_key(bt)
        ctx.upload_keyswitch_key(ks)
        rl = rng.integers(0, P.Q, (3, 2 * P.N), dtype=np.uint64)
        rl[0] = P.Q - 1
        d = dev(torch, rl)
        out = torch.zeros((3, P.n + 1), dtype=torch.int64, device="cuda")
        ctx.lwe_keyswitch_async(d.data_ptr(), 3, out.data_ptr())
        ctx.sync()
        assert np.array_equal(out.cpu().numpy().view(np.uint64), np.stack([o.lwe_keyswitch(r, ks) for r in rl]))
        for count in (1, 100, 400):
            ct = F.LWE_encrypt(P, 5 + count, lsk, rng.integers(0, 2, 2 * count, dtype=np.uint8))
            g = rng.integers(0, 6, count).astype(np.int32)
            got = ctx.eval_bootstrap_batch(ct[:count], ct[count:], g)
            idx = np.unique(np.linspace(0, count - 1, 12).astype(int))
            want, _ = o.eval_bootstrap_batch(ct[:count][idx], ct[count:][idx], g[idx], bt, ks)
            assert np.array_equal(got[idx], want), count
