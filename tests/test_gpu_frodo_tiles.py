"""FrodoKEM tensor-core batches with scratch for all, some or none of their operand tiles: keypair, encaps,
decaps and decaps of tampered ciphertexts against the dot-product form on every instance and the CPU oracle on a
sample.  The number of instances with tiles is computed beside each case, so that a case that stops
reaching its path fails."""
import os

import numpy as np
import pytest
import torch

import dpcrypto_b200 as d

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 8
TILES = 2162688  # bytes of tiles an instance
SCRATCH = 15680 * 2 + 24 + 24 + 4 + 200  # and of scratch, each array rounded up to 256 bytes


def _tiles(n, nbytes):
    """Instances of a batch of n that get tiles in an arena of nbytes (two product CTAs an SM)."""
    wave = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    room = max(0, (nbytes - n * SCRATCH - 5 * 256) // TILES)
    most = n if n <= 1024 else wave + n % wave
    if room >= most:
        return most
    if room < n % wave or 1024 < n <= 4096:
        return 0
    return n % wave + (room - n % wave) // wave * wave


def _case(engine, scheme, n):
    kc = torch.empty((n, 64), dtype=torch.uint8, device="cuda")
    ec = torch.empty((n, 24), dtype=torch.uint8, device="cuda")
    engine.coins(n, 64, "tiles-kp", out=kc)
    engine.coins(n, 24, "tiles-enc", out=ec)
    pk, sk = engine.keypair(scheme, kc, d.FORM_DP4A)
    ct, ss = engine.enc(scheme, pk, ec, d.FORM_DP4A)
    bad = ct.clone()
    i = torch.arange(0, n, 2, device="cuda")
    bad[i, (i * 7919 + 15743) % 15744] ^= 32
    rej = engine.dec(scheme, bad, sk, d.FORM_DP4A)
    return kc, ec, pk, sk, ct, ss, bad, rej


def _check(eng, oracle, scheme, case):
    kc, ec, pk, sk, ct, ss, bad, rej = case
    got_k, got_e = eng.keypair(scheme, kc), eng.enc(scheme, pk, ec)
    assert torch.equal(got_k[0], pk) and torch.equal(got_k[1], sk)
    assert torch.equal(got_e[0], ct) and torch.equal(got_e[1], ss)
    assert torch.equal(eng.dec(scheme, ct, sk), ss) and torch.equal(eng.dec(scheme, bad, sk), rej)
    same = (rej == ss).all(dim=1)
    assert not same[::2].any() and same[1::2].all()
    n = kc.shape[0]
    idx = sorted({0, n // 2, n - 1})
    h = lambda t: np.ascontiguousarray(t[idx].cpu().numpy())  # noqa: E731
    pk_o, sk_o = oracle.keypair(scheme, h(kc), threads=THREADS)
    ct_o, ss_o = oracle.enc(scheme, pk_o, h(ec), threads=THREADS)
    assert (h(got_k[0]) == pk_o).all() and (h(got_k[1]) == sk_o).all()
    assert (h(got_e[0]) == ct_o).all() and (h(got_e[1]) == ss_o).all()
    assert (h(rej) == oracle.dec(scheme, h(bad), sk_o, threads=THREADS)).all()


@pytest.mark.parametrize("scheme,n,mib,tiles", [
    (d.FRODO976, 7, 4, 0), (d.FRODO976, 40, 72, 0), (d.FRODO976, 40, 100, 40),
    (d.FRODO976AES, 40, 72, 0), (d.FRODO976, 300, 64, 4), (d.FRODO976AES, 300, 64, 4), (d.FRODO976, 300, 16, 0),
    (d.FRODO976, 600, 720, 304), (d.FRODO976, 1100, 200, 0), (d.FRODO976AES, 1100, 1200, 508),
    (d.FRODO976, 4500, 320, 60)])
def test_reserved_arena(engine, oracle, scheme, n, mib, tiles):
    assert _tiles(n, mib << 20) == tiles
    case = _case(engine, scheme, n)
    torch.cuda.synchronize()
    with d.Engine(0) as eng:
        eng.reserve(mib << 20)
        _check(eng, oracle, scheme, case)


@pytest.mark.parametrize("scheme,n", [(d.FRODO976, 24), (d.FRODO976, 25), (d.FRODO976AES, 24)])
def test_product_blocks(engine, oracle, scheme, n):
    """Two column blocks a product CTA up to 24 instances, four above."""
    _check(engine, oracle, scheme, _case(engine, scheme, n))


@pytest.mark.parametrize("scheme", [d.FRODO976, d.FRODO976AES])
def test_budget_without_tiles(engine, oracle, scheme):
    """A budget of 4 MiB: half of it is scratch, chunks of 66 and 34, no room for tiles; host buffers too."""
    n = 100
    chunk = (2 << 20) // (SCRATCH + 80 + 32)
    assert chunk == 66 and _tiles(chunk, 4 << 20) == 0
    case = _case(engine, scheme, n)
    torch.cuda.synchronize()
    with d.Engine(0, hbm_budget=4 << 20) as eng:
        _check(eng, oracle, scheme, case)
        kc, ec, pk, sk, ct, ss, bad, rej = (t.cpu().numpy() for t in case)
        got_k, got_e = eng.keypair(scheme, kc), eng.enc(scheme, pk, ec)
        assert (got_k[0] == pk).all() and (got_k[1] == sk).all() and (got_e[0] == ct).all() and (got_e[1] == ss).all()
        assert (eng.dec(scheme, bad, sk) == rej).all()


@pytest.mark.parametrize("scheme,n", [(d.FRODO976, 1025), (d.FRODO976AES, 1025)])
def test_profiled_batch_without_tiles(engine, oracle, scheme, n):
    case = _case(engine, scheme, n)
    with d.Engine(0) as eng:
        eng.profile(True)
        _check(eng, oracle, scheme, case)
        assert len(eng.stage_times()) == 4 and all(t > 0 for t in eng.stage_times())


def test_profiled_stages_without_tiles(engine, oracle):
    """profile(2): a batch that would be generated whole runs without tiles, all of A in the product stage (with
    tiles that stage is a pass of MMAs, a few per cent of the call)."""
    case = _case(engine, d.FRODO976, 64)
    kc, ec, pk, sk, ct, ss, bad, rej = case
    with d.Engine(0) as eng:
        share = {}
        for mode in (True, 2):
            eng.profile(mode)
            _check(eng, oracle, d.FRODO976, case)
            eng.enc(d.FRODO976, pk, ec)
            t = eng.stage_times()
            assert len(t) == 3
            share[mode] = t[1] / sum(t)
    assert share[True] < 0.15 and share[2] > 0.25, share
