"""Timed cases of the library: the work its users have it do, through the
package's public entry points.

The operators' inputs are uniform field elements, as the benchmark's are;
points are uniform multiples of the generator.  Results that are points are
taken to affine form (or, for proofs, to the 256-byte wire form): that is the
form a user stores or sends, and the canonical one, because a Jacobian triple
is only one of many for its point.

Kinds of a case:
  ntt    in-place transforms of `count` vectors of 2^log_n elements
  msm    one multi-scalar multiplication, over plain bases or over a
         shifted-copy table; `bits` is the share of scalars that are 0 or 1
  spmv   A z, B z, C z of a synthetic circuit
  prove  Groth16 proofs: the synthetic circuit in standard mode, or the
         matrix-product circuit in the reference-compatible mode
  batch  many MSMs and NTTs of uneven sizes as one captured plan
"""
import math

import numpy as np
import torch

from liblightzk_b200 import _capi, autotune, groth16, msm, ntt, synth
from liblightzk_b200.batch import BatchPlan

# the moduli are BN254's
R_FR = 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001
FR_TOP = R_FR >> 192          # top 64-bit limb; a smaller top limb makes any element canonical


def listed():
    return [
        # a short transform by itself: the smallest call a program makes often
        {"name": "ntt_fwd_2e12", "kind": "ntt", "log_n": 12, "direction": ntt.FORWARD, "count": 1},
        # the transform of a prover's three vectors at 2^17 constraints
        {"name": "ntt_inv_3x2e17", "kind": "ntt", "log_n": 17, "direction": ntt.INVERSE, "count": 3},
        # the coset transform at the benchmark's size
        {"name": "ntt_coset_fwd_2e20", "kind": "ntt", "log_n": 20, "direction": ntt.COSET_FORWARD, "count": 1},
        # the largest single transform of the benchmark, with its coset factors
        {"name": "ntt_coset_inv_2e24", "kind": "ntt", "log_n": 24, "direction": ntt.COSET_INVERSE, "count": 1},
        # commitment to a short vector over bases seen for the first time
        {"name": "msm_g1_plain_1000", "kind": "msm", "group": 1, "n": 1000, "table": False, "bits": 0.0},
        # the benchmark's plain MSM
        {"name": "msm_g1_plain_2e16", "kind": "msm", "group": 1, "n": 1 << 16, "table": False, "bits": 0.0},
        # a fixed key's query over its table, ragged, near the benchmark's 2^20
        {"name": "msm_g1_table_1000003", "kind": "msm", "group": 1, "n": 1000003, "table": True, "bits": 0.0},
        # the same in G2, at a middle size
        {"name": "msm_g2_table_200003", "kind": "msm", "group": 2, "n": 200003, "table": True, "bits": 0.0},
        # constraint evaluation at the benchmark's size
        {"name": "spmv_2e20", "kind": "spmv", "log_m": 20},
        # one proof of a small circuit: latency
        {"name": "prove_2e12", "kind": "prove", "circuit": "synthetic", "log_m": 12},
        # one proof of the benchmark's circuit
        {"name": "prove_2e20", "kind": "prove", "circuit": "synthetic", "log_m": 20},
        # the batched operators: uneven MSMs over fixed bases beside transforms
        {"name": "batch_24msm_12ntt", "kind": "batch", "n_msm": 24, "n_ntt": 12, "msm_log": 18, "ntt_log": 20, "shape": 5},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ntt", "ntt", "msm", "msm", "msm", "msm", "spmv", "prove", "prove", "batch"])
    if kind == "ntt":
        log_n = rng.randint(8, 23)
        return {"kind": kind, "log_n": log_n, "direction": rng.randint(0, 3),
                "count": rng.randint(1, min(9, 1 << (23 - log_n)))}
    if kind == "msm":
        # half of a real witness is often zeros and ones
        group = rng.choice([1, 1, 2])
        return {"kind": kind, "group": group, "n": _log_uniform(rng, 300, 1 << (20 if group == 1 else 19)),
                "table": rng.random() < 0.5, "bits": rng.choice([0.0, 0.0, 0.5])}
    if kind == "spmv":
        return {"kind": kind, "log_m": rng.randint(10, 20)}
    if kind == "prove":
        if rng.random() < 0.4:
            return {"kind": kind, "circuit": "matmul", "p": _log_uniform(rng, 9, 63)}
        return {"kind": kind, "circuit": "synthetic", "log_m": rng.randint(9, 18)}
    return {"kind": kind, "n_msm": rng.randint(2, 24), "n_ntt": rng.randint(0, 12), "msm_log": rng.randint(13, 18),
            "ntt_log": rng.randint(13, 20), "shape": rng.randint(0, 1 << 30)}


_tuned = False


def _start():
    """what a program does once: install the packaged tuning table"""
    global _tuned
    if not _tuned:
        autotune.load_default()
        _tuned = True


def _fr(n, gen):
    """n uniform Fr elements in Montgomery form: random limbs, the top one
    below the modulus's"""
    x = torch.randint(-(1 << 63), (1 << 63) - 1, (n, 4), dtype=torch.int64, device="cuda", generator=gen)
    x[:, 3] = torch.randint(0, FR_TOP, (n,), dtype=torch.int64, device="cuda", generator=gen)
    return x


def _scalars(n, bits, gen):
    s = _fr(n, gen)
    if bits:
        one = torch.from_numpy(synth.FR_ONE.view(np.int64)).cuda()
        pick = torch.rand(n, device="cuda", generator=gen)
        s[pick < bits / 2] = 0
        s[(pick >= bits / 2) & (pick < bits)] = one
    return s


def _circuit(case, seed):
    if case["circuit"] == "matmul":
        return synth.MatMulCircuit(case["p"])
    return synth.Circuit(case["log_m"], seed=seed)


def prepare(case, seed):
    _start()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    st = {"case": case}
    if kind == "ntt":
        ntt.prepare(case["log_n"])
        st["data"] = _fr(case["count"] << case["log_n"], gen)
    elif kind == "msm":
        g, n = case["group"], case["n"]
        st["scalars"] = _scalars(n, case["bits"], gen)
        st["bases"] = synth.fixed_base(g, _fr(n, gen))
        if case["table"]:
            c = st["c"] = msm.autotune_window(g, n, precomputed=True)
            st["table"] = msm.precompute(g, st["bases"], c)
            del st["bases"]
    elif kind == "spmv":
        st["circuit"] = c = synth.Circuit(case["log_m"], seed=seed)
        st["mats"] = [m.desc() for m in c.mats]
        st["z"] = _fr(c.n_vars, gen)
        st["out"] = [torch.empty((c.M, 4), dtype=torch.int64, device="cuda") for _ in range(3)]
    elif kind == "prove":
        c = _circuit(case, seed)
        mode = groth16.REFERENCE if case["circuit"] == "matmul" else groth16.STANDARD
        st["prover"] = groth16.Prover(c, synth.ProvingKey(c, seed=seed + 1), mode=mode)
        st["z"] = c.witness(seed + 2)
        st["r"], st["s"] = _fr(2, gen).cpu().numpy().view(np.uint64)
    else:
        rng = np.random.default_rng(case["shape"])
        sizes = np.rint(2.0 ** rng.uniform(10, case["msm_log"], case["n_msm"])).astype(np.int64)
        logs = rng.integers(10, case["ntt_log"] + 1, case["n_ntt"])
        dirs = rng.integers(0, 4, case["n_ntt"])
        st["jac"] = torch.empty((case["n_msm"], 3, 4), dtype=torch.int64, device="cuda")
        msms = [(_fr(int(n), gen), synth.fixed_base(1, _fr(int(n), gen)), st["jac"][i]) for i, n in enumerate(sizes)]
        st["vecs"] = [_fr(1 << int(k), gen) for k in logs]
        ntts = [(v, int(k), int(d)) for v, k, d in zip(st["vecs"], logs, dirs)]
        st["plan"] = BatchPlan(1, msms=msms, ntts=ntts, fixed_bases=True)
        st["stream"] = torch.cuda.Stream()
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ntt":
        if case["count"] == 1:
            return ntt.ntt(state["data"], case["log_n"], case["direction"])
        return ntt.ntt_batch(state["data"], case["log_n"], case["count"], 1 << case["log_n"], case["direction"])
    if kind == "msm":
        g, n = case["group"], case["n"]
        if case["table"]:
            c = state["c"]
            jac = msm.msm_precomputed(g, state["scalars"], state["table"], c, msm.windows_for(c), n)
        else:
            jac = msm.msm(g, state["scalars"], state["bases"])
        return msm.to_affine(g, jac[None])
    if kind == "spmv":
        ntt.spmv3(*state["mats"], state["z"], *state["out"])
        return state["out"]
    if kind == "prove":
        return groth16.to_wire(state["prover"].prove(state["z"], state["r"], state["s"]))
    s = state["stream"]
    state["plan"].run(use_graph=True, stream=s)
    with torch.cuda.stream(s):
        return [msm.to_affine(1, state["jac"], stream=s)] + state["vecs"]


# Work: bytes each input and output once; operations as 32-bit multiply-add
# steps, 264 to a Montgomery product of the 254-bit fields (8 x 8 limbs, low
# and high halves, and the reduction).
_PRODUCT = 264.0


def _msm_work(group, n, table):
    """an addition to each bucket (10 products of Fq, 30 for Fq2) for every
    window of every scalar; a window is about as wide as a fixed base's table
    of this size allows"""
    c = max(4, min(17, int(math.log2(max(n, 2))) - 3))
    adds = n * math.ceil(255 / c)
    point = 64 * group
    copies = math.ceil(255 / c) if table else 1
    return n * 32 + n * copies * point, adds * (10 if group == 1 else 30) * _PRODUCT


def _ntt_work(log_n, direction, count):
    n = count << log_n
    extra = n if direction != ntt.FORWARD else 0
    return 2 * n * 32, (n / 2 * log_n + extra) * _PRODUCT


def _prove_shape(case):
    """(constraints, variables, entries of the three matrices, those to multiply by)"""
    if case["circuit"] == "matmul":
        p = case["p"]
        m = 1 << (p ** 3 + p * p - 1).bit_length()
        return m, 1 + 3 * p * p + p ** 3, 4 * p ** 3 + 2 * p * p, 0
    m = 1 << case["log_m"]
    return m, m + 4098, 6 * m, 3 * m


def work(case):
    kind = case["kind"]
    if kind == "ntt":
        b, f = _ntt_work(case["log_n"], case["direction"], case["count"])
    elif kind == "msm":
        b, f = _msm_work(case["group"], case["n"], case["table"])
        f *= 1 - case["bits"]
    elif kind == "spmv":
        m = 1 << case["log_m"]
        b, f = 6 * m * 36 + 3 * m * 4 + (m + 4098) * 32 + 3 * m * 32, 3 * m * _PRODUCT
    elif kind == "prove":
        m, n, nnz, mul = _prove_shape(case)
        b, f = nnz * 36 + n * 32, mul * _PRODUCT
        log_m = m.bit_length() - 1
        ref = case["circuit"] == "matmul"
        for group, k in ((1, n), (1, n), (1, n + m), (2, n)):
            x, y = _msm_work(group, k, True)
            b, f = b + x, f + y
        big = log_m + 1 if ref else log_m
        for d, k, c in ((ntt.INVERSE, log_m, 3), (ntt.FORWARD, big, 3), (ntt.INVERSE, big, 1)):
            f += _ntt_work(k, d, c)[1]
    else:
        rng = np.random.default_rng(case["shape"])
        sizes = np.rint(2.0 ** rng.uniform(10, case["msm_log"], case["n_msm"]))
        logs = rng.integers(10, case["ntt_log"] + 1, case["n_ntt"])
        parts = [_msm_work(1, int(n), True) for n in sizes] + [_ntt_work(int(k), ntt.INVERSE, 1) for k in logs]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    return {"bytes": float(b), "flops": float(f)}


def _to_ints(t):
    return [int.from_bytes(x.tobytes(), "little") for x in t.cpu().numpy()]


def _from_ints(v):
    a = np.frombuffer(b"".join(x.to_bytes(32, "little") for x in v), dtype=np.int64)
    return torch.from_numpy(a.reshape(-1, 4).copy())


def _transform(a, log_n, direction):
    """X_k = sum_j a_j w^(jk) on plain integers; the Montgomery factor of
    the elements passes through, since the transform is linear"""
    n = 1 << log_n
    w = pow(5, (R_FR - 1) >> log_n, R_FR)
    if direction == ntt.COSET_FORWARD:
        f = 1
        for i in range(n):
            a[i] = a[i] * f % R_FR
            f = f * 5 % R_FR
    if direction in (ntt.INVERSE, ntt.COSET_INVERSE):
        w = pow(w, -1, R_FR)
    a = [a[int(format(i, "0%db" % log_n)[::-1], 2)] for i in range(n)] if log_n else a
    half = 1
    while half < n:
        step = pow(w, n // (2 * half), R_FR)
        tw = [1]
        for _ in range(half - 1):
            tw.append(tw[-1] * step % R_FR)
        for s in range(0, n, 2 * half):
            for j in range(half):
                u, v = a[s + j], a[s + j + half] * tw[j] % R_FR
                a[s + j], a[s + j + half] = (u + v) % R_FR, (u - v) % R_FR
        half *= 2
    if direction in (ntt.INVERSE, ntt.COSET_INVERSE):
        f, g = pow(n, -1, R_FR), pow(5, -1, R_FR) if direction == ntt.COSET_INVERSE else 1
        for i in range(n):
            a[i] = a[i] * f % R_FR
            f = f * g % R_FR
    return a


def exact(case, seed):
    """transforms small enough for Python's integers; the other results are
    whole numbers too, and are compared as such"""
    if case["kind"] != "ntt" or case["count"] << case["log_n"] > 1 << 18:
        return None
    data, n = prepare(case, seed)["data"], 1 << case["log_n"]
    return torch.cat([_from_ints(_transform(_to_ints(data[i * n:(i + 1) * n]), case["log_n"], case["direction"]))
                      for i in range(case["count"])])
