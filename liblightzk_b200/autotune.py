"""Measured autotuner for the library's tuning table (lzk_tune_set).

Per size class 2^log_n it times candidates on the device (CUDA events,
seeded random inputs, median of a few runs) and installs the fastest:

  window  Pippenger window width of plain-base MSMs (the cost model's
          width and its neighbours)
  chunk   sorted bucket entries one accumulation thread adds (8 to 128)
  run     buckets per lane run in the bucket-reduction tiles (1 to 16)
  ntt     elements per block of an NTT pass, i.e. how a transform's stages
          split into passes (256, 512, 1024, 2048)
  table_*  window width, chunk and run of MSMs over shifted-copy tables
          (provers, batch plans with fixed bases)

The sweeps reach from 2^6 to 2^21 points (2^24 elements); `fill_edges` gives
the size classes beyond them the values of the nearest one measured.

Every autotuned MSM, batch plan and prover made afterwards uses the table
(a prover or plan reads it when it is created).  `save` / `load` keep a
table as JSON, so a tuned table can be reused without re-timing.
"""
import json
import os

import numpy as np
import torch

from . import _capi, msm, ntt, synth

# measured tables shipped with the package, by GPU name
DEFAULT_TABLES = {"B200": os.path.join(os.path.dirname(os.path.abspath(__file__)), "tuning", "b200.json")}

WINDOW, CHUNK, RUN, NTT_BLOCK, TABLE_WINDOW, TABLE_CHUNK, TABLE_RUN = range(7)
KNOBS = {"window": WINDOW, "chunk": CHUNK, "run": RUN, "ntt": NTT_BLOCK, "table_window": TABLE_WINDOW,
         "table_chunk": TABLE_CHUNK, "table_run": TABLE_RUN}
# candidates of the sweeps: short chunks and runs are for lists that leave the
# device idle, long ones for lists that fill it several times
CHUNKS, RUNS, BLOCKS = (8, 16, 32, 64, 128), (1, 2, 4, 8, 16), (256, 512, 1024, 2048)
# size classes the sweeps of a whole table cover, by group: plain MSMs, table
# MSMs, and transforms
PLAIN_CLASSES = {1: range(6, 22), 2: range(8, 21)}
TABLE_CLASSES = {1: range(8, 21), 2: range(8, 21)}
NTT_CLASSES = range(10, 25)
# plain G1 widths hold up to this class: at 2^22 to 2^25 points the width of 2^21
# is within 1 % of the best; from 2^26 on the cost model's is better (200 instead
# of 205 ms), and at 2^28 narrow ones make more entries than can be numbered
PLAIN_WIDTH_TOP = 25


def _time(fn, reps):
    ts = []
    for _ in range(reps + 1):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        torch.cuda.synchronize()
        ts.append(a.elapsed_time(b))
    return float(np.median(ts[1:]))


def set_value(knob, group, log_n, value):
    _capi.call("lzk_tune_set", KNOBS[knob], group, log_n, value)


def get_value(knob, group, log_n):
    return int(_capi.lib().lzk_tune_get(KNOBS[knob], group, log_n))


def tune(group=1, log_ns=range(10, 21), spread=2, reps=3, seed=11, install=True):
    """window widths only: {log_n: (best_c, {c: ms})}"""
    table = {}
    top = max(log_ns)
    sc_all = synth.random_fr(1 << top, seed, 90)
    bases_all = synth.fixed_base(group, synth.random_fr(1 << top, seed, 91))
    for lg in log_ns:
        n = 1 << lg
        set_value("window", group, lg, 0)      # model value as the centre
        c0 = msm.autotune_window(group, n)
        res = {}
        for c in range(max(2, c0 - spread), min(22, c0 + spread) + 1):
            res[c] = _time(lambda c=c: msm.msm(group, sc_all[:n], bases_all[:n], window_bits=c), reps)
        best = min(res, key=res.get)
        table[lg] = (best, res)
        if install:
            set_value("window", group, lg, best)
    return table


def _best(res):
    """the fastest (width, run, chunk), the times by width and run (with the
    best chunk) and by chunk (at the best width and run)"""
    c, r, v = min(res, key=res.get)
    pairs = {}
    for (x, y, _), ms in res.items():
        pairs[(x, y)] = min(ms, pairs.get((x, y), ms))
    return c, r, v, pairs, {z: ms for (x, y, z), ms in res.items() if (x, y) == (c, r)}


def tune_msm(group=1, log_ns=None, spread=2, reps=3, seed=11, chunks=CHUNKS, runs=RUNS):
    """per size class: window width, reduction run and accumulation chunk
    together (the run sets how much each bucket costs and a short chunk fills
    the device with few entries, which both move the best width); installs
    them and returns
    {log_n: {"window": best_c, "run": best_run, "chunk": best_chunk,
             "ms": {"c,run": ms}, "chunk_ms": {chunk: ms}}}"""
    out = {}
    log_ns = PLAIN_CLASSES[group] if log_ns is None else log_ns
    top = max(log_ns)
    sc_all = synth.random_fr(1 << top, seed, 90)
    bases_all = synth.fixed_base(group, synth.random_fr(1 << top, seed, 91))
    for lg in log_ns:
        n = 1 << lg
        s, b = sc_all[:n], bases_all[:n]
        for k in ("window", "chunk", "run"):
            set_value(k, group, lg, 0)
        c0 = msm.autotune_window(group, n)
        res = {}
        for c in range(max(2, c0 - spread), min(22, c0 + spread) + 1):
            for r in runs:
                set_value("run", group, lg, r)
                for v in chunks:
                    set_value("chunk", group, lg, v)
                    res[(c, r, v)] = _time(lambda c=c: msm.msm(group, s, b, window_bits=c), reps)
        c_best, r_best, ch_best, res, cres = _best(res)
        set_value("window", group, lg, c_best)
        set_value("run", group, lg, r_best)
        set_value("chunk", group, lg, ch_best)
        out[lg] = {"window": c_best, "run": r_best, "chunk": ch_best,
                   "ms": {f"{c},{r}": v for (c, r), v in res.items()}, "chunk_ms": cres}
    return out


def tune_msm_table(group=1, log_ns=None, spread=(4, 2), reps=3, seed=11, runs=RUNS, chunks=CHUNKS):
    """window width, reduction run and chunk together, of an MSM over a
    shifted-copy table, per size class, timing one MSM of 2^log_n points
    (the table of each width built outside the timing; widths from
    spread[0] below the cost model's to spread[1] above); installs the best
    and returns {log_n: {"window", "run", "chunk", "ms": {"c,run": ms},
    "chunk_ms": {chunk: ms}}}"""
    out = {}
    log_ns = TABLE_CLASSES[group] if log_ns is None else log_ns
    top = max(log_ns)
    sc_all = synth.random_fr(1 << top, seed, 94)
    bases_all = synth.fixed_base(group, synth.random_fr(1 << top, seed, 95))
    for lg in log_ns:
        n = 1 << lg
        s, b = sc_all[:n], bases_all[:n]
        for knob in ("table_window", "table_run", "table_chunk"):
            set_value(knob, group, lg, 0)
        c0 = msm.autotune_window(group, n, precomputed=True)
        res = {}
        # the model leans to wide windows (it undercounts the bucket
        # reduction), so the candidates reach further below it than above
        for c in range(max(4, c0 - spread[0]), min(20, c0 + spread[1]) + 1):
            w = msm.windows_for(c)
            tab = msm.precompute(group, b, c, w, n)
            for r in runs:
                set_value("table_run", group, lg, r)
                for v in chunks:
                    set_value("table_chunk", group, lg, v)
                    res[(c, r, v)] = _time(lambda c=c, w=w: msm.msm_precomputed(group, s, tab, c, w, n), reps)
            del tab
        c_best, r_best, ch_best, res, cres = _best(res)
        set_value("table_window", group, lg, c_best)
        set_value("table_run", group, lg, r_best)
        set_value("table_chunk", group, lg, ch_best)
        out[lg] = {"window": c_best, "run": r_best, "chunk": ch_best,
                   "ms": {f"{c},{r}": v for (c, r), v in res.items()}, "chunk_ms": cres}
    return out


def tune_ntt(log_ns=NTT_CLASSES, reps=3, seed=12, blocks=BLOCKS, direction=ntt.COSET_FORWARD):
    """NTT block size per transform size; installs the fastest and returns
    {log_n: (best, {block: ms})}"""
    out = {}
    for lg in log_ns:
        x = synth.random_fr(1 << lg, seed, 92)
        ntt.prepare(lg)
        res = {}
        for v in blocks:
            set_value("ntt", 0, lg, v)
            res[v] = _time(lambda: ntt.ntt(x, lg, direction), reps)
        best = min(res, key=res.get)
        set_value("ntt", 0, lg, best)
        out[lg] = (best, res)
    return out


def tune_prover(circuit, pk, mode=0, window_bits=0, chunks=CHUNKS[:4], runs=RUNS, proofs=8, seed=13):
    """accumulation chunk and reduction run of a Groth16 prover's own MSMs
    (shifted-table MSMs over the circuit's variables, the L + H concatenation
    and the G2 query), chosen by timing whole proofs; installs the best
    pair for those size classes and returns {(chunk, run): ms per proof}"""
    from . import device, groth16
    z = circuit.witness(seed)
    rs = device.to_host(synth.random_fr(2, seed, 93))
    nl = circuit.n_vars - circuit.n_public - 1
    classes = {1: {int(np.ceil(np.log2(circuit.n_vars))), int(np.ceil(np.log2(nl + circuit.M - 1)))},
               2: {int(np.ceil(np.log2(circuit.n_vars)))}}

    def install(chunk, run):
        for g, lgs in classes.items():
            for lg in lgs:
                set_value("table_chunk", g, lg, chunk)
                set_value("table_run", g, lg, run)

    res = {}
    for chunk in chunks:
        for run in runs:
            install(chunk, run)
            p = groth16.Prover(circuit, pk, mode=mode, window_bits=window_bits)
            res[(chunk, run)] = _time(lambda: [p.prove(z, rs[0], rs[1]) for _ in range(proofs)], 2) / proofs
            p.close()
    best = min(res, key=res.get)
    install(*best)
    return res


def fill_edges():
    """give the size classes outside the sweeps the values of the nearest class
    in them; table widths above stay unset (the cost model), plain G1 ones from
    2^26 on too (PLAIN_WIDTH_TOP), and so do all of G2 above"""
    def copy(knob, group, classes, top):
        for lg in range(33):
            if lg < classes[0]:
                set_value(knob, group, lg, get_value(knob, group, classes[0]))
            elif lg > classes[-1]:
                set_value(knob, group, lg, get_value(knob, group, classes[-1]) if lg <= top else 0)
    for g in (1, 2):
        copy("window", g, PLAIN_CLASSES[g], PLAIN_WIDTH_TOP if g == 1 else 0)
        for knob in ("chunk", "run"):
            copy(knob, g, PLAIN_CLASSES[g], 32 if g == 1 else 0)
        for knob in ("table_window", "table_chunk", "table_run"):
            for lg in range(TABLE_CLASSES[g][0]):
                set_value(knob, g, lg, get_value(knob, g, TABLE_CLASSES[g][0]))
    copy("ntt", 0, NTT_CLASSES, 32)


def load_default():
    """install the packaged table measured on this GPU model, if there is
    one; returns its path or None"""
    name = torch.cuda.get_device_name()
    for key, path in DEFAULT_TABLES.items():
        if key in name and os.path.exists(path):
            load(path)
            return path
    return None


def current(groups=(1, 2), log_ns=range(0, 33)):
    """the installed table as a JSON-able dict of non-default entries"""
    t = {"msm": {}, "ntt": {}}
    for g in groups:
        t["msm"][str(g)] = {k: {str(lg): get_value(k, g, lg) for lg in log_ns}
                            for k in ("window", "chunk", "run", "table_window", "table_chunk", "table_run")}
    t["ntt"] = {str(lg): get_value("ntt", 0, lg) for lg in log_ns}
    return t


def save(path, table=None):
    with open(path, "w") as f:
        json.dump(table or current(), f, indent=1, sort_keys=True)


def load(path):
    """install a table written by save()"""
    t = json.load(open(path))
    for g, knobs in t.get("msm", {}).items():
        for k, vals in knobs.items():
            for lg, v in vals.items():
                set_value(k, int(g), int(lg), int(v))
    for lg, v in t.get("ntt", {}).items():
        set_value("ntt", 0, int(lg), int(v))
