"""Two contexts used by two host threads: kernels that both launch take different
amounts of shared memory (n, digitG), and neither thread's launches may depend on
what the other asked for last."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(F, torch, preset, n, bg):
    """A context, one gate's device buffers and its output by a call of its own."""
    P = F.params_preset(preset)
    P.n, P.BG_bits, P.digitG = n, bg, 0
    F.derive(P)
    lsk, rsk = F.LWE_secretkey(P, 1), F.RLWE_secretkey(P, 2)
    ctx = F.Context(P, 0)
    ctx.upload_bootstrap_key(F.bootstrap_key(P, 3, lsk, rsk))
    ctx.upload_keyswitch_key(F.keyswitch_key(P, 4, rsk, lsk))
    ct = F.LWE_encrypt(P, 5, lsk, np.array([0, 1], dtype=np.uint8))
    d = torch.from_numpy(ct.view(np.int64)).cuda()
    gate = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.zeros_like(d[:1])
    args = (d.data_ptr(), d[1:].data_ptr(), gate.data_ptr(), 1, out.data_ptr())
    torch.cuda.synchronize()
    ctx.bootstrap_async(*args)
    ctx.sync()
    return ctx, args, out, out.clone(), (d, gate)


@pytest.mark.parametrize("preset,sets", [(0, [(5, 7), (60, 7)]), (1, [(2, 9), (2, 14)])])
def test_two_threads(F, cuda_ok, preset, sets):
    torch = cuda_ok
    made = [make(F, torch, preset, n, bg) for n, bg in sets]
    errors = []

    def work(ctx, args):
        try:
            for i in range(3000):
                ctx.bootstrap_async(*args)
                if i % 50 == 49:
                    ctx.sync()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(m[0], m[1])) for m in made]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for ctx, _, out, want, _ in made:
        assert torch.equal(out, want)
        ctx.close()
