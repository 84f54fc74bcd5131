"""The work a prover built on this library has it do, as cases to be timed.

Each family is one entry point of the C ABI (or one short sequence that is always called together), over the sizes
that the tests, the benchmark and its batched / served mixes use:

  commit   Ajtai commitments (kappa = 16) of n_vec digit matrices: device buffers with the small-digit promise
           (form "small"), device buffers of any int8 digits ("any"), or host buffers ("host"); any m, odd ones too
  ccs      one Pi_CCS RoundOracle's whole life: created from host buffers, every row and Ajtai round evaluated at
           0..6 and folded as a sum-check driver does, the ME outputs, destroyed
  mem      one Twist / Shout time-lane RoundOracle's whole life on columns in device memory
  taddr    one Twist address-lane RoundOracle's whole life on columns in device memory
  rlc_dec  the Pi_RLC mix of `count` digit matrices and the balanced split of the result into 12 planes
  fold     one steady-state fold step (k = 13) of a shard with one Twist memory and one Shout table

All arithmetic is exact (F_q, K = F_q^2, small integers): every output is a whole number.
"""
import ctypes

import numpy as np
import torch

from nightstream_b200 import gpu, synth

KAPPA, D, K_RHO, ELL_D, D_SC = 16, 54, 12, 6, 6

_ctx = None
_fold_ccs = {}


def context():
    """The process's context (one device, one stream), kept as a prover keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = gpu.Context(0)
    return _ctx


def listed():
    return [
        # the MCS commitment of the smallest shard: latency
        {"name": "commit_mcs_1k", "family": "commit", "form": "small", "n_vec": 1, "m": 1 << 10},
        # the 12 DEC children of the benchmarked shard in one call
        {"name": "commit_dec_64k", "family": "commit", "form": "small", "n_vec": 12, "m": 1 << 16},
        # digits of a larger base, a size that is no power of two, a ragged vector count
        {"name": "commit_any_10k", "family": "commit", "form": "any", "n_vec": 5, "m": 10006},
        # SModuleHomomorphism::commit as the reference's prover calls it, host buffers, an odd column count
        {"name": "commit_host_odd", "family": "commit", "form": "host", "n_vec": 1, "m": 5001},
        # Pi_CCS of the benchmarked shard (MCS witness and 12 children) driven round by round
        {"name": "ccs_64k", "family": "ccs", "ell": 16, "k": 13},
        # Pi_CCS of the smallest shard's first step
        {"name": "ccs_1k", "family": "ccs", "ell": 10, "k": 1},
        # Twist read check: 2^16 time rows, 2^14 of them active, 2^12 cells
        {"name": "mem_read_64k", "family": "mem", "kind": gpu.MEM_TWIST_READ, "ell": 16, "ell_addr": 12, "active": 1 << 14},
        # bitness of a Twist instance's columns (2 * 10 address bits and a gate) on a short trace
        {"name": "mem_bits_4k", "family": "mem", "kind": gpu.MEM_BITNESS, "ell": 12, "ell_addr": 10, "active": 1000},
        # Twist read check over the addresses of a large shard's 2^14 trace steps
        {"name": "taddr_16k", "family": "taddr", "kind": 0, "ell": 14, "ell_addr": 16, "active": 1 << 14},
        # Pi_RLC / Pi_DEC witness work of a mid-size shard through host buffers
        {"name": "rlc_dec_16k", "family": "rlc_dec", "count": 13, "m": 1 << 14},
        # the benchmarked fold step: 2^16 constraints, 1024 trace steps, Twist 2^12 cells, Shout 2^16 entries
        {"name": "fold_64k", "family": "fold", "ell": 16, "steps": 1024, "twist": 12, "shout": 16},
        # a large shard: 2^18 constraints, 4096 trace steps, Twist 2^14 cells, Shout 2^18 entries
        {"name": "fold_256k", "family": "fold", "ell": 18, "steps": 4096, "twist": 14, "shout": 18},
    ]


def _log_int(rng, lo, hi):
    return int(round(2 ** rng.uniform(np.log2(lo), np.log2(hi))))


def draw(rng):
    family = rng.choice(["commit", "commit", "ccs", "mem", "mem", "taddr", "rlc_dec", "fold"])
    if family == "commit":
        form = rng.choice(["small", "small", "any", "host"])
        m = _log_int(rng, 1 << 9, 1 << 14 if form == "host" else 1 << 16)
        if form != "host" and rng.random() < 0.75:
            m += m & 1  # most witnesses have an even column count
        elif m % 2:
            m = min(m, 1 << 14 | 1)
        return {"family": family, "form": form, "n_vec": rng.randint(1, 3) if form == "host" else rng.randint(1, 13), "m": m}
    if family == "ccs":
        return {"family": family, "ell": rng.randint(6, 16), "k": rng.choice([1, 2, 5, 13, 13, 13])}
    if family == "mem":
        ell = rng.randint(8, 16)
        return {"family": family, "kind": rng.randint(0, 6), "ell": ell, "ell_addr": rng.randint(4, 14),
                "active": _log_int(rng, 40, 1 << min(ell, 14))}
    if family == "taddr":
        ell = rng.randint(8, 14)
        return {"family": family, "kind": rng.randint(0, 1), "ell": ell, "ell_addr": rng.randint(6, 16),
                "active": _log_int(rng, 40, 1 << ell)}
    if family == "rlc_dec":
        return {"family": family, "count": rng.randint(2, 13), "m": _log_int(rng, 1 << 8, 1 << 15)}
    ell = rng.randint(12, 16)
    # the trace has to leave the constraints room: (twist, shout) bus columns times steps stay under half the witness
    return {"family": family, "ell": ell, "steps": _log_int(rng, 16, (1 << ell) // 96), "twist": rng.randint(6, 10),
            "shout": rng.randint(6, 12)}


# ---- inputs --------------------------------------------------------------------

def _rng(case, seed):
    return np.random.default_rng([seed, sum(map(ord, case["family"]))])


def _trace(rng, ell, ell_addr, active):
    """Time columns (int64 K pairs, on the host) of a memory trace: per step at most one read and one write, 70 %
    stride-4 sequential and 30 % uniform addresses, 32-bit values, increments against the current memory."""
    L, P = 1 << ell, 1 << ell_addr
    mem = rng.integers(0, 1 << 32, size=P).tolist()
    start = list(mem)
    cols = {n: np.zeros(L, np.uint64) for n in ("has_read", "has_write", "ra", "wa", "rv", "wv", "inc")}
    seq, uni = rng.random(active) < 0.7, rng.integers(0, P, size=active).tolist()
    step, vals = rng.integers(0, 2, size=active).tolist(), rng.integers(0, 1 << 32, size=active).tolist()
    reads, writes = rng.random(active) < 0.9, rng.random(active) < 0.8
    pos = 0
    q = 0xFFFFFFFF00000001
    for t in range(active):
        if seq[t]:
            pos = (pos + 4) % P
        a = pos if seq[t] else uni[t]
        if reads[t]:
            cols["has_read"][t], cols["ra"][t], cols["rv"][t] = 1, a, mem[a]
        if writes[t]:
            w = (a + step[t]) % P
            cols["has_write"][t], cols["wa"][t], cols["wv"][t] = 1, w, vals[t]
            cols["inc"][t] = (vals[t] - mem[w]) % q
            mem[w] = vals[t]
    return cols, start


def _bits(v, n):
    return [(v >> np.uint64(b)) & np.uint64(1) for b in range(n)]


def _device_cols(cols):
    """Base-field columns as K columns [n_cols][2^ell][2] in device memory."""
    c = np.zeros((len(cols), cols[0].size, 2), np.uint64)
    for i, v in enumerate(cols):
        c[i, :, 0] = v
    return torch.from_numpy(c.view(np.int64)).cuda()


def _fold_circuit(case):
    """The circuit of a fold case, made once: its constraints avoid the witness's bus tail, so every trace of the
    same shape satisfies it."""
    key = (case["ell"], case["steps"], case["twist"], case["shout"])
    if key not in _fold_ccs:
        m = 1 << case["ell"]
        base = m - (case["shout"] + 2 + 2 * case["twist"] + 5) * case["steps"]
        z = np.random.default_rng(case["ell"]).integers(0, 1 << 32, size=m, dtype=np.uint64)
        z[0] = 1
        _fold_ccs.clear()
        _fold_ccs[key] = (*synth.make_r1cs(case["ell"], 11, z=z, max_col=base), base)
    return _fold_ccs[key]


def _public_parameters(m):
    """The public parameters of column count m: one per m in a process, so every state of that m shares them."""
    context().pp_generate(bytes((m + i) % 256 for i in range(32)), KAPPA, m)


def prepare(case, seed):
    ctx, rng, family = context(), _rng(case, seed), case["family"]
    s = {"case": case}
    if family == "commit":
        n_vec, m = case["n_vec"], case["m"]
        _public_parameters(m)
        lim = 128 if case["form"] == "any" else 2
        g = torch.Generator(device="cuda").manual_seed(seed)
        digits = torch.randint(1 - lim, lim, (n_vec, D, m), dtype=torch.int8, device="cuda", generator=g)
        if case["form"] == "host":
            s["digits"] = digits.cpu().numpy()
        else:
            s["digits"] = digits
            s["out"] = torch.zeros((n_vec, KAPPA, D), dtype=torch.int64, device="cuda")
    elif family == "ccs":
        ell, k = case["ell"], case["k"]
        ccs, z = synth.make_r1cs(ell, seed)
        digits = [rng.integers(-1, 2, size=(D, 1 << ell), dtype=np.int8) for _ in range(k - 1)]
        s["args"] = (ccs, np.stack([ctx.decomp_b2(z)] + digits), 2, synth.uniform_k(rng, ELL_D),
                     synth.uniform_k(rng, ELL_D), synth.uniform_k(rng, ell), synth.uniform_k(rng, 1)[0],
                     synth.uniform_k(rng, ell) if k > 1 else None, ELL_D, ell, D_SC)
        s["xs"] = np.array([[x, 0] for x in range(D_SC + 1)], np.uint64)
        s["chals"] = synth.uniform_k(rng, ell + ELL_D)
    elif family in ("mem", "taddr"):
        ell, A, kind = case["ell"], case["ell_addr"], case["kind"]
        c, start = _trace(rng, ell, A, case["active"])
        read = [c["has_read"], c["rv"], *_bits(c["ra"], A), c["has_write"], c["inc"], *_bits(c["wa"], A)]
        write = [c["has_write"], c["wv"], c["inc"], *_bits(c["wa"], A)]
        if family == "taddr":
            s["cols"] = _device_cols(write if kind else read)
            s["init_addr"] = np.arange(1 << A, dtype=np.uint64)
            s["init_val"] = np.stack([np.array(start, np.uint64), np.zeros(1 << A, np.uint64)], axis=1)
            s["chals"] = synth.uniform_k(rng, A)
        else:
            cols = {gpu.MEM_SHOUT_VALUE: [c["has_read"], c["rv"]],
                    gpu.MEM_SHOUT_ADAPTER: [c["has_read"], *_bits(c["ra"], A)],
                    gpu.MEM_BITNESS: [c["has_read"], *_bits(c["ra"], A), *_bits(c["wa"], A)],
                    gpu.MEM_TWIST_READ: read, gpu.MEM_TWIST_WRITE: write,
                    gpu.MEM_VAL_EVAL: [c["has_write"], c["inc"], *_bits(c["wa"], A)],
                    gpu.MEM_TOTAL_INC: [c["has_write"], c["inc"], *_bits(c["wa"], A)]}[kind]
            s["cols"] = _device_cols(cols)
            s["r_addr"], s["init"] = synth.uniform_k(rng, A), synth.uniform_k(rng, 1)
            s["weights"] = synth.uniform_k(rng, len(cols))
            s["chals"] = synth.uniform_k(rng, ell)
        s["point"] = synth.uniform_k(rng, ell)
    elif family == "rlc_dec":
        s["rho"] = rng.integers(-2, 3, size=(case["count"], D), dtype=np.int8)
        s["digits"] = rng.integers(-1, 2, size=(case["count"], D, case["m"]), dtype=np.int8)
    else:
        ccs, z, base = _fold_circuit(case)
        buses, mem, inits = synth.memory_trace_chunks(2, case["steps"], case["shout"], case["twist"], seed)
        _public_parameters(z.size)
        s["z"] = []
        for bus in buses:
            zc = z.copy()
            zc[base:] = bus.reshape(-1)
            s["z"].append(zc)
        s["inits"], s["chunk"] = inits, 1
        s["shard"] = gpu.Shard(ctx, ccs, mem=mem)
        s["shard"].fold_step(s["z"][0])  # the first step has no children yet; the timed ones do
    torch.cuda.synchronize()
    return s


# ---- one pass ------------------------------------------------------------------

def _k(a):
    return a.view(np.int64)


def _oracle(ctx, create, close, evals, fold, rounds, degree, chals):
    """A RoundOracle driven as a sum-check driver does: every round at 0..degree, the challenge folded in, and the
    final value."""
    h = ctypes.c_void_p()
    create(ctypes.byref(h))
    xs = np.array([[x, 0] for x in range(degree(h) + 1)], np.uint64)
    ys = np.empty((rounds + 1, *xs.shape), np.uint64)
    for i in range(rounds + 1):
        ctx.check(evals(h, xs.ctypes.data, len(xs), ys[i].ctypes.data))
        if i < rounds:
            ctx.check(fold(h, chals[i].ctypes.data))
    close(h)
    return _k(ys)


def run(s):
    ctx, case = context(), s["case"]
    family, lib = case["family"], ctx.lib
    if family == "commit":
        if case["form"] == "host":
            ctx.kappa = KAPPA
            return _k(ctx.commit(s["digits"]))
        ctx.commit_device(s["digits"].data_ptr(), case["n_vec"], case["m"], s["out"].data_ptr(),
                          small_digits=case["form"] == "small")
        return s["out"]
    if family == "ccs":
        o = gpu.GpuCcsOracle(ctx, *s["args"])
        ys = np.empty((len(s["chals"]), *s["xs"].shape), np.uint64)
        for i, r in enumerate(s["chals"]):
            ys[i] = o.evals_at(s["xs"])
            o.fold(r)
        y, y_scalars = o.me_outputs()
        o.close()
        return {"rounds": _k(ys), "y": _k(y), "y_scalars": _k(y_scalars)}
    if family == "mem":
        claim, kind, A = np.empty(2, np.uint64), case["kind"], case["ell_addr"]
        no_addr = kind in (gpu.MEM_SHOUT_VALUE, gpu.MEM_BITNESS)
        ys = _oracle(ctx, lambda h: ctx.check(lib.neo_gpu_mem_oracle_create_device(
            ctx.h, kind, case["ell"], s["point"].ctypes.data, 0 if no_addr else A,
            None if no_addr else s["r_addr"].ctypes.data, s["init"].ctypes.data, len(s["cols"]), s["cols"].data_ptr(),
            s["weights"].ctypes.data, claim.ctypes.data, h)),
            lib.neo_gpu_mem_oracle_destroy, lib.neo_gpu_mem_oracle_evals, lib.neo_gpu_mem_oracle_fold, case["ell"],
            lib.neo_gpu_mem_oracle_degree_bound, s["chals"])
        return {"rounds": ys, "claim": _k(claim)}
    if family == "taddr":
        return _oracle(ctx, lambda h: ctx.check(lib.neo_gpu_twist_addr_create_device(
            ctx.h, case["kind"], case["ell"], s["point"].ctypes.data, case["ell_addr"], len(s["init_addr"]),
            s["init_addr"].ctypes.data, s["init_val"].ctypes.data, s["cols"].data_ptr(), h)),
            lib.neo_gpu_twist_addr_destroy, lib.neo_gpu_twist_addr_evals, lib.neo_gpu_twist_addr_fold,
            case["ell_addr"], lib.neo_gpu_twist_addr_degree_bound, s["chals"])
    if family == "rlc_dec":
        mix = ctx.rlc_mix(s["rho"], s["digits"])
        planes, nonzero = ctx.split_b(mix, K_RHO, 2)
        return {"mix": mix, "planes": planes, "nonzero": nonzero}
    c = s["chunk"]
    s["chunk"] = 1 - c
    s["shard"].set_twist_init(0, s["inits"][c][0])
    proof = s["shard"].fold_step(s["z"][c])
    return {"proof": _k(proof), "transcript": _k(s["shard"].transcript_state())}


# ---- what a pass cannot do without ------------------------------------------------

def _commit_work(n_vec, m):
    """Each digit and each public parameter once; kappa d^2 products of an 8-byte coefficient and a digit a column."""
    return n_vec * D * m + KAPPA * D * m * 8 + n_vec * KAPPA * D * 8, 2 * 8 * n_vec * KAPPA * D * D * m


def work(case):
    family = case["family"]
    if family == "commit":
        b, f = _commit_work(case["n_vec"], case["m"])
    elif family == "ccs":
        n = 1 << case["ell"]
        # the digits and the matrices once; a field product (32 operations) for each nonzero, and a few for each row
        # of each of the small tables over all rounds
        b = case["k"] * D * n + 9 * n * 12 + 4 * 54 * 16 * case["k"]
        f = 32 * (2 * 9 * n + 60 * n) + 2 * case["k"] * D * n
    elif family in ("mem", "taddr"):
        L, A = 1 << case["ell"], case["ell_addr"]
        if family == "mem":
            n_cols = {0: 2, 1: 1 + A, 2: 1 + 2 * A, 3: 4 + 2 * A, 4: 3 + A, 5: 2 + A, 6: 2 + A}[case["kind"]]
            f = 96 * 2 * (n_cols + 1) * case["active"]  # folding each column's active rows
        else:
            n_cols = 3 + A if case["kind"] else 4 + 2 * A
            f = 96 * 4 * A * case["active"] + 96 * (1 << A)
        b = n_cols * L * 16 + ((16 << A) if family == "taddr" else 0)
    elif family == "rlc_dec":
        n, m = case["count"], case["m"]
        b, f = n * D * m + 4 * D * m + K_RHO * D * m, 2 * n * D * D * m + 3 * K_RHO * D * m
    else:
        m = 1 << case["ell"]
        cb, cf = _commit_work(2 * K_RHO + 1, m)
        oracle = work({"family": "ccs", "ell": case["ell"], "k": K_RHO + 1})
        mixes = 2 * (K_RHO + 3) * D * D * m
        b, f = cb + 8 * m + oracle["bytes"] + 4 * K_RHO * D * m, cf + oracle["flops"] + mixes
    return {"bytes": int(b), "flops": int(f)}


def exact(case, seed):
    """Every output is a whole number (F_q words, digits): equal or wrong, with no 64-bit value to be near to."""
    return None
