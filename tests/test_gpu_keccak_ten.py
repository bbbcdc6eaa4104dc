"""Keccak-f[1600] on ten lanes per state (keccak10.cuh), which most sponge chains run, against the CPU oracle's
permutation: random and edge states, one, two and three states in the last warp, and a dependent chain."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _oracle(oracle, states, perms):
    lib, out = oracle.lib(), states.copy()
    for s in range(states.shape[0]):
        row = np.ascontiguousarray(out[s])
        for _ in range(perms):
            lib.oracle_keccak_f1600(row.ctypes.data)
        out[s] = row
    return out


def _run(engine, states, perms):
    got = engine.keccak_lanes(10, torch.from_numpy(states.view(np.int64)).cuda(), perms)
    return got.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("n,perms", [(1, 0), (1, 1), (2, 1), (3, 24), (4, 3), (31, 2), (600, 2), (601, 1)])
def test_matches_oracle(engine, oracle, n, perms):
    rng = np.random.default_rng(n * 10 + perms)
    states = rng.integers(0, 2**64, size=(n, 25), dtype=np.uint64)
    states[0] = 0
    if n > 1:
        states[1] = np.uint64(0xFFFFFFFFFFFFFFFF)
    assert (_run(engine, states, perms) == _oracle(oracle, states, perms)).all()


def test_single_bits(engine, oracle):
    """Every bit of every lane alone: each (half, rotation, lane) path of the bit-interleaved form."""
    bits = np.zeros((1600, 25), np.uint64)
    for b in range(1600):
        bits[b, b // 64] = np.uint64(1) << np.uint64(b % 64)
    assert (_run(engine, bits, 0) == bits).all()
    assert (_run(engine, bits, 1) == _oracle(oracle, bits, 1)).all()


def test_probe(engine):
    assert engine.probe_keccak_chain(10, 7, 4) > 0
