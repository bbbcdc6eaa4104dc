"""FrodoKEM batches whose A is generated ahead of its use (tensor-core form, a key per
instance): every byte against the dp4a form on every instance and against the CPU oracle on a
sample, at the sizes where the split of a batch changes (one instance, the columns of a product
split over one, two and four CTAs, the largest batch generated whole, the largest on ten lanes and
the largest on lane pairs, each with the size after it)."""
import os

import numpy as np
import pytest
import torch

import dpcrypto_b200 as d

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 8


def _sample(n):
    return sorted({0, n // 2, n - 1})


@pytest.mark.parametrize("scheme,n", [(s, n) for s in (d.FRODO976, d.FRODO976AES)
                                      for n in (1, 3, 49, 50, 98, 99, 297)] +
                         [(d.FRODO976, n) for n in (444, 445, 1024, 1025, 1100, 4096, 4097, 9472, 9473)])
def test_ahead_equals_dp4a_and_oracle(engine, oracle, scheme, n):
    kc = torch.empty((n, 64), dtype=torch.uint8, device="cuda")
    ec = torch.empty((n, 24), dtype=torch.uint8, device="cuda")
    engine.coins(n, 64, "ahead-kp", out=kc)
    engine.coins(n, 24, "ahead-enc", out=ec)
    pk, sk = engine.keypair(scheme, kc, d.FORM_TC)
    pk4, sk4 = engine.keypair(scheme, kc, d.FORM_DP4A)
    assert torch.equal(pk, pk4) and torch.equal(sk, sk4)
    ct, ss = engine.enc(scheme, pk, ec, d.FORM_TC)
    ct4, ss4 = engine.enc(scheme, pk, ec, d.FORM_DP4A)
    assert torch.equal(ct, ct4) and torch.equal(ss, ss4)
    assert torch.equal(engine.dec(scheme, ct, sk, d.FORM_TC), ss)
    bad = ct.clone()
    pos = (torch.arange(n, device="cuda") * 7919) % bad.shape[1]
    pos[0] = bad.shape[1] - 1  # the last byte of C, then positions over all of ct
    bad[torch.arange(n, device="cuda"), pos] ^= 1
    rej = engine.dec(scheme, bad, sk, d.FORM_TC)
    assert torch.equal(rej, engine.dec(scheme, bad, sk, d.FORM_DP4A))
    assert not (rej == ss).all(dim=1).any()
    idx = _sample(n)
    h = lambda t: np.ascontiguousarray(t[idx].cpu().numpy())  # noqa: E731
    pk_o, sk_o = oracle.keypair(scheme, h(kc), threads=THREADS)
    assert (h(pk) == pk_o).all() and (h(sk) == sk_o).all()
    ct_o, ss_o = oracle.enc(scheme, pk_o, h(ec), threads=THREADS)
    assert (h(ct) == ct_o).all() and (h(ss) == ss_o).all()
    assert (h(rej) == oracle.dec(scheme, h(bad), sk_o, threads=THREADS)).all()


@pytest.mark.parametrize("mib", [65, 72, 160])
def test_small_budgets(oracle, mib):
    """An arena budget that holds no operand tiles, a few, and more than the batch needs."""
    n = 40
    kc = oracle.coins(n, 64, "ahead-b")
    ec = oracle.coins(n, 24, "ahead-b")
    with d.Engine(0, hbm_budget=mib << 20) as eng:
        pk, sk = eng.keypair(d.FRODO976, kc)
        ct, ss = eng.enc(d.FRODO976, pk, ec)
        assert (eng.dec(d.FRODO976, ct, sk) == ss).all()
    pk_o, sk_o = oracle.keypair(0, kc, threads=THREADS)
    assert (pk == pk_o).all() and (sk == sk_o).all()
    ct_o, ss_o = oracle.enc(0, pk_o, ec, threads=THREADS)
    assert (ct == ct_o).all() and (ss == ss_o).all()
