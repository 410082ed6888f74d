"""The work that users of this framework have it do, as timed cases.

A case names one call (or one short sequence of calls) through the package's
public entry points:

  gates    a batch of independent gate bootstraps, ciphertexts in device memory
           (Context.bootstrap_async)
  host     the same through host arrays (Context.eval_bootstrap_batch): what a
           program written against the reference runtime's fixed-width calls does
  server   one PSI equality query through the serving loop (Server.submit / poll)
  expand   expand_RLWE of one packed RLWE into N RLWEs
  cmux     one level of a CMUX tree: `count` pairs selected by one RGSW
  psi      the reference's PSI query at N = 2048: homo_expand, a CMUX tree over a
           database of 2^levels RLWEs, an RLWE blind rotation

`preset` is the parameter set: 0 (N = 1024, 27-bit Q, digitG 4), 1 (N = 2048,
54-bit Q, digitG 6), 2 (N = 1024, 27-bit Q, digitG 3).

A program that evaluates gates holds one evaluation key for as long as it runs:
the keys are made from fixed seeds and stay in one context per parameter set,
and the ciphertexts come from the seed of prepare(). All outputs are whole
numbers (ciphertext words), so exact() has nothing to add.
"""
import functools
import importlib

import numpy as np
import torch

F = importlib.import_module("3rd_gen_fhe_acc_gb300")

GATES = (F.OR, F.AND, F.NOR, F.NAND, F.XOR, F.XNOR)


def listed():
    return [
        # latency of one gate: a program whose next gate needs this one's result
        {"name": "lone_gate_n1024", "kind": "gates", "preset": 0, "count": 1},
        # the widest fixed-width call of the reference's FPGA backend (10 gates), host arrays in and out
        {"name": "host_10_gates_n1024", "kind": "host", "preset": 0, "count": 10},
        # a level of a small circuit (less than one gate per SM), the CPU app's parameter set
        {"name": "gates_96_digit3", "kind": "gates", "preset": 2, "count": 96},
        # a ragged serving round of a few gates per SM
        {"name": "gates_333_n1024", "kind": "gates", "preset": 0, "count": 333},
        # one level of a wide circuit
        {"name": "gates_1000_n1024", "kind": "gates", "preset": 0, "count": 1000},
        # the headline batch: 4096 independent gates
        {"name": "gates_4096_n1024", "kind": "gates", "preset": 0, "count": 4096},
        # one PSI equality query (16 items of 32 bits: 1008 gates in 6 levels) through the server
        {"name": "server_query_16_items", "kind": "server", "preset": 0, "count": 16},
        # the wide parameter set: one gate, a small level, a ragged round, the large batch
        {"name": "lone_gate_n2048", "kind": "gates", "preset": 1, "count": 1},
        {"name": "gates_100_n2048", "kind": "gates", "preset": 1, "count": 100},
        {"name": "gates_700_n2048", "kind": "gates", "preset": 1, "count": 700},
        {"name": "gates_2048_n2048", "kind": "gates", "preset": 1, "count": 2048},
        # the reference's PSI query: 128 database entries
        {"name": "psi_query_n2048", "kind": "psi", "preset": 1, "count": 7},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["gates", "gates", "gates", "host", "server", "expand", "cmux", "psi"])
    if kind == "gates":
        preset = rng.choice([0, 0, 1, 2])
        return {"kind": kind, "preset": preset, "count": _log_uniform(rng, 1, 2048 if preset == 1 else 4096)}
    if kind == "host":
        return {"kind": kind, "preset": rng.choice([0, 2]), "count": _log_uniform(rng, 1, 2000)}
    if kind == "server":
        return {"kind": kind, "preset": 0, "count": _log_uniform(rng, 1, 64)}
    if kind == "expand":
        # the flag picks the device or a caller's own stream: an option of every asynchronous entry point
        return {"kind": kind, "preset": rng.choice([0, 1]), "count": 1, "own_stream": rng.random() < 0.5}
    if kind == "cmux":
        return {"kind": kind, "preset": rng.choice([0, 1]), "count": _log_uniform(rng, 1, 1024)}
    return {"kind": kind, "preset": 1, "count": rng.randint(1, 9)}


@functools.lru_cache(maxsize=None)
def _context(preset):
    """One context with resident keys per parameter set, and its LWE secret key."""
    p = F.params_preset(preset)
    lsk = F.LWE_secretkey(p, 11 + preset)
    rsk = F.RLWE_secretkey(p, 21 + preset)
    ctx = F.Context(p, 0)
    ctx.upload_bootstrap_key(F.bootstrap_key(p, 31 + preset, lsk, rsk))
    ctx.upload_keyswitch_key(F.keyswitch_key(p, 41 + preset, rsk, lsk))
    ctx.upload_subs_key(F.substitute_key(p, 51 + preset, rsk))
    return p, ctx, lsk


def _device(words):
    return torch.from_numpy(np.ascontiguousarray(words).view(np.int64)).cuda()


def _uniform(seed, shape, q):
    """Words uniform mod Q, as the polynomials of fresh ciphertexts are."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, q, shape, dtype=torch.int64, device="cuda", generator=g)


def prepare(case, seed):
    kind, count = case["kind"], case["count"]
    p, ctx, lsk = _context(case["preset"])
    rw, gw = 2 * p.N, p.digitG * 4 * p.N
    s = {"kind": kind, "count": count, "p": p, "ctx": ctx, "rw": rw, "gw": gw}
    rng = np.random.default_rng(seed)
    if kind in ("gates", "host"):
        ct = F.LWE_encrypt(p, 1000 + seed, lsk, rng.integers(0, 2, 2 * count, dtype=np.uint8))
        gates = rng.choice(GATES, count).astype(np.int32)
        if kind == "host":
            s.update(c1=ct[:count], c2=ct[count:], gates=gates)
        else:
            s.update(c1=_device(ct[:count]), c2=_device(ct[count:]), gates=torch.from_numpy(gates).cuda())
            s["out"] = torch.zeros_like(s["c1"])
    elif kind == "server":
        s["inputs"] = F.LWE_encrypt(p, 1000 + seed, lsk, rng.integers(0, 2, 32 * (1 + count), dtype=np.uint8))
        s["circuit"] = F.psi_equality_circuit(count)
        s["server"] = F.Server(ctx, max_batch=2048, pool_ciphertexts=1 << 16)
    elif kind == "expand":
        s["packed"] = _uniform(seed, (rw,), p.Q)
        s["out"] = torch.zeros((p.N, rw), dtype=torch.int64, device="cuda")
        if case.get("own_stream"):
            s["stream"] = torch.cuda.Stream()
    elif kind == "cmux":
        s["pairs"] = _uniform(seed, (2 * count, rw), p.Q)
        s["select"] = _uniform(seed + 1, (gw,), p.Q)
        s["out"] = torch.zeros((count, rw), dtype=torch.int64, device="cuda")
    else:
        s["packed"] = _uniform(seed, (p.digitG, rw), p.Q)
        s["enc_neg_s"] = _uniform(seed + 1, (gw,), p.Q)
        s["database"] = _uniform(seed + 2, (1 << count, rw), p.Q)
        s["rgsw"] = torch.zeros((p.N, gw), dtype=torch.int64, device="cuda")
        s["levels"] = [torch.zeros(((1 << count) // 2, rw), dtype=torch.int64, device="cuda") for _ in range(2)]
        s["out"] = torch.zeros(rw, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    return s


def run(s):
    kind, ctx, count, rw, gw = s["kind"], s["ctx"], s["count"], s["rw"], s["gw"]
    here = torch.cuda.current_stream()
    st = here.cuda_stream
    if kind == "gates":
        ctx.bootstrap_async(s["c1"].data_ptr(), s["c2"].data_ptr(), s["gates"].data_ptr(), count,
                            s["out"].data_ptr(), stream=st)
        return s["out"]
    if kind == "host":
        return ctx.eval_bootstrap_batch(s["c1"], s["c2"], s["gates"])
    if kind == "server":
        _, out = s["server"].submit(s["inputs"], *s["circuit"])
        while not s["server"].poll(timeout_ms=100):
            pass
        return out
    if kind == "expand":
        own = s.get("stream", here)
        if own is not here:
            own.wait_stream(here)
        ctx.expand_RLWE(s["packed"].data_ptr(), s["out"].data_ptr(), stream=own.cuda_stream)
        if own is not here:
            here.wait_stream(own)
        return s["out"]
    if kind == "cmux":
        p0 = s["pairs"].data_ptr()
        ctx.CMUX(p0, p0 + 8 * rw, s["select"].data_ptr(), s["out"].data_ptr(), count, in_stride=2 * rw, stream=st)
        return s["out"]
    ctx.homo_expand(s["packed"].data_ptr(), s["enc_neg_s"].data_ptr(), s["rgsw"].data_ptr(), stream=st)
    src, n, level = s["database"], 1 << count, s["p"].N.bit_length() - 1
    while n > 1:   # entry k of the next level: pair (2k, 2k + 1) selected by the level's RGSW
        dst = s["levels"][level & 1]
        ctx.CMUX(src.data_ptr(), src.data_ptr() + 8 * rw, s["rgsw"].data_ptr() + 8 * gw * level, dst.data_ptr(),
                 n // 2, in_stride=2 * rw, stream=st)
        src, n, level = dst, n // 2, level + 1
    ctx.blind_rotate_RLWE(src.data_ptr(), s["rgsw"].data_ptr(), False, s["out"].data_ptr(), 1, stream=st)
    return s["out"]


def work(case):
    """Bytes: evaluation-key words that `count` ciphertexts select, read once (4 bytes each for a 27-bit Q, 8 for a
    54-bit one), inputs and outputs. Operations: two per modular multiplication of the transforms and products (an
    N-point transform: N/2 log2 N; a product of one RLWE and one RGSW: 2 + 2 digitG transforms, 4 digitG N
    multiplications)."""
    kind, count, p = case["kind"], case["count"], F.params_preset(case["preset"])
    N, dG, logN = p.N, p.digitG, p.N.bit_length() - 1
    word = 4 if p.Q < 1 << 32 else 8
    ntt = N // 2 * logN
    product = (2 + 2 * dG) * ntt + 4 * dG * N
    rlwe, rgsw = 2 * N, 4 * dG * N
    if kind in ("gates", "host", "server"):
        gates = 63 * count if kind == "server" else count
        steps = p.n * p.digitR * (p.Br - 1) / p.Br
        keys = p.n * p.digitR * (p.Br - 1) * (1 - (1 - 1 / p.Br) ** gates) * rgsw
        rows = p.digitKS * N * p.Bks * (1 - (1 - 1 / p.Bks) ** gates) * (p.n + 1)
        inputs = 32 * (1 + count) + count if kind == "server" else 3 * count
        return {"bytes": word * (keys + rows) + 8 * inputs * (p.n + 1),
                "flops": 2 * gates * (steps * product + 2 * ntt + p.digitKS * N * (p.n + 1) / 2)}
    subs = logN * p.digitKS_R * rlwe
    expand = (N - 1) * ((3 + p.digitKS_R) * ntt + (2 * p.digitKS_R + 2) * N)
    if kind == "expand":
        return {"bytes": word * subs + 8 * (rlwe + N * rlwe), "flops": 2 * expand}
    if kind == "cmux":
        return {"bytes": 8 * (3 * count * rlwe + rgsw), "flops": 2 * count * product}
    cmux = (1 << count) - 1 + logN
    return {"bytes": 8 * (dG * rlwe + rgsw + (1 << count) * rlwe + rlwe + N * rgsw) + word * subs,
            "flops": 2 * (dG * expand + (dG * N + cmux) * product)}
