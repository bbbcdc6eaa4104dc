"""Saber batches on both sides of the rules that depend on level and form: how a call's kernels follow one
another (FireSaber), where decaps leave the lane pairs (LightSaber).  Every byte of all forms against one another and of a sample against the CPU oracle."""
import os

import numpy as np
import pytest
import torch

import dpcrypto_b200 as d

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 8


def _check(engine, oracle, scheme, n, forms):
    z = d.sizes(scheme)
    kc = torch.empty((n, z["kp_coins"]), dtype=torch.uint8, device="cuda")
    ec = torch.empty((n, z["enc_coins"]), dtype=torch.uint8, device="cuda")
    engine.coins(n, z["kp_coins"], "rule-kp", out=kc)
    engine.coins(n, z["enc_coins"], "rule-enc", out=ec)
    res = []
    for form in forms:
        pk, sk = engine.keypair(scheme, kc, form)
        ct, ss = engine.enc(scheme, pk, ec, form)
        bad = ct.clone()
        bad[torch.arange(n, device="cuda"), (torch.arange(n, device="cuda") * 7919) % z["ct"]] ^= 4
        back, rej = engine.dec(scheme, ct, sk, form), engine.dec(scheme, bad, sk, form)
        assert torch.equal(back, ss) and not (rej == ss).all(dim=1).any()
        res.append((pk, sk, ct, ss, bad, rej))
    for r in res[1:]:
        for a, b in zip(res[0], r):
            assert torch.equal(a, b)
    idx = sorted({0, n // 2, n - 1})
    h = lambda t: np.ascontiguousarray(t[idx].cpu().numpy())  # noqa: E731
    pk, sk, ct, ss, bad, rej = (h(t) for t in res[0])
    pk_o, sk_o = oracle.keypair(scheme, h(kc), threads=THREADS)
    ct_o, ss_o = oracle.enc(scheme, pk_o, h(ec), threads=THREADS)
    assert (pk == pk_o).all() and (sk == sk_o).all() and (ct == ct_o).all() and (ss == ss_o).all()
    assert (rej == oracle.dec(scheme, bad, sk_o, threads=THREADS)).all()


@pytest.mark.parametrize("n", [100, 101, 148, 149, 350, 351, 444, 445, 512, 513])
def test_following_kernels(engine, oracle, n):
    _check(engine, oracle, d.FIRESABER, n, (d.FORM_TC, d.FORM_DP4A, d.FORM_INT32))


@pytest.mark.parametrize("n", [4736, 4737])
def test_lightsaber_decaps_pairs(engine, oracle, n):
    _check(engine, oracle, d.LIGHTSABER, n, (d.FORM_TC, d.FORM_DP4A))
