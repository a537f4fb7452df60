"""Scalars over the endomorphism of G1 (csrc/glv.cuh): plain MSMs and the
prover's variable-base products with scalars at the edges of the split (0, 1,
r - 1, lambda, and those whose lattice coordinates lie next to a half)."""
import random

import numpy as np
import pytest

from helpers import bases, same_point
from oracle import FR

R = 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001
LAMBDA = 0xB3C4D79D41A917585BFC41088D8DAAA78B17EA66B99C90DD
A, B = 0x89D3256894D213E3, 0x6F4D8248EEB859FC8211BBEB7D4F1128

pytestmark = pytest.mark.gpu


def _edges(count):
    rng = random.Random(1)
    ks = [0, 1, 2, R - 1, R - 2, R // 2, R // 2 + 1, LAMBDA, R - LAMBDA, LAMBDA + 1]
    while len(ks) < count:
        for m in (A, B):
            ks.append(((2 * rng.randrange(m) + 1) * R // (2 * m) + rng.randrange(-1, 3)) % R)
    return ks[:count]


def _mont(orc, ks):
    return orc.to_mont(FR, np.array([[k >> (64 * i) & (1 << 64) - 1 for i in range(4)] for k in ks], np.uint64))


@pytest.mark.parametrize("n,c", [(1, 2), (10, 3), (333, 7), (501, 13), (501, 16)])
def test_split_edges(cuda, orc, rng_state, n, c):
    from liblightzk_b200 import device, msm
    s, b = _mont(orc, _edges(n)), bases(orc, 1, n, rng_state)
    b[n // 3] = 0
    got = msm.msm(1, device.to_device(s), device.to_device(b), window_bits=c)
    assert same_point(orc, 1, device.to_host(got), orc.msm(1, s, b))


def test_proofs_with_edge_randomness(cuda, orc):
    from liblightzk_b200 import device, groth16, synth
    circ = synth.Circuit(6, seed=9, n_public=1, n_free=8, block=16)
    pk, z, h = synth.ProvingKey(circ, seed=10), circ.witness(11), device.to_host
    keys = {"a_query": h(pk.a), "b1_query": h(pk.b1), "b2_query": h(pk.b2), "l_query": h(pk.l), "h_query": h(pk.h),
            "alpha1": h(pk.alpha1), "beta1": h(pk.beta1), "delta1": h(pk.delta1), "beta2": h(pk.beta2),
            "delta2": h(pk.delta2)}
    prover = groth16.Prover(circ, pk, window_bits=6)
    vals = _mont(orc, _edges(14))
    for i in range(0, 14, 2):
        r, s = vals[i], vals[i + 1]
        got = groth16.split_proof(prover.prove(z, r, s))
        want = orc.groth16_prove([m.host() for m in circ.mats], circ.M, circ.n_vars, circ.n_public, circ.log_m, keys,
                                 h(z), r, s, groth16.STANDARD)
        for g, a, b in zip((1, 2, 1), got, want):
            assert same_point(orc, g, a, b)
