"""Saber batches across the rules that choose a stage's layout: lanes per state of the sponges
(a warp, ten lanes, a pair, one), XOF bytes left as bit-interleaved halves between prologue and
product, GenMatrix beside the inner product.  Every byte of the tensor-core form against the
INT32 form and of both against the CPU oracle on a sample; sizes with partial warps and blocks."""
import os

import numpy as np
import pytest
import torch

import dpcrypto_b200 as d

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 8
BIG = 1 << 30
LAYOUTS = {"warp": dict(saber_warp_max=BIG, saber_finish_warp_max=BIG),
           "ten": dict(saber_warp_max=0, saber_five_max=BIG, saber_finish_warp_max=0, saber_finish_five_max=BIG),
           "pair": dict(saber_warp_max=0, saber_five_max=0, saber_finish_warp_max=0, saber_finish_five_max=0,
                        saber_pair_max=BIG),
           "one": dict(saber_warp_max=0, saber_five_max=0, saber_finish_warp_max=0, saber_finish_five_max=0,
                       saber_pair_max=0)}


def _run(engine, oracle, scheme, n):
    z = d.sizes(scheme)
    kc = torch.empty((n, z["kp_coins"]), dtype=torch.uint8, device="cuda")
    ec = torch.empty((n, z["enc_coins"]), dtype=torch.uint8, device="cuda")
    engine.coins(n, z["kp_coins"], "lay-kp", out=kc)
    engine.coins(n, z["enc_coins"], "lay-enc", out=ec)
    res = {}
    for form in (d.FORM_TC, d.FORM_INT32):
        pk, sk = engine.keypair(scheme, kc, form)
        ct, ss = engine.enc(scheme, pk, ec, form)
        bad = ct.clone()
        pos = (torch.arange(n, device="cuda") * 7919 + z["ct"] - 1) % z["ct"]  # the last byte first
        bad[torch.arange(n, device="cuda"), pos] ^= 128
        back, rej = engine.dec(scheme, ct, sk, form), engine.dec(scheme, bad, sk, form)
        assert torch.equal(back, ss) and not (rej == ss).all(dim=1).any()
        res[form] = (pk, sk, ct, ss, bad, rej)
    for a, b in zip(res[d.FORM_TC], res[d.FORM_INT32]):
        assert torch.equal(a, b)
    idx = sorted({0, n // 3, n - 1})
    h = lambda t: np.ascontiguousarray(t[idx].cpu().numpy())  # noqa: E731
    pk, sk, ct, ss, bad, rej = (h(t) for t in res[d.FORM_TC])
    pk_o, sk_o = oracle.keypair(scheme, h(kc), threads=THREADS)
    ct_o, ss_o = oracle.enc(scheme, pk_o, h(ec), threads=THREADS)
    assert (pk == pk_o).all() and (sk == sk_o).all() and (ct == ct_o).all() and (ss == ss_o).all()
    assert (rej == oracle.dec(scheme, bad, sk_o, threads=THREADS)).all()


@pytest.mark.parametrize("scheme", [d.LIGHTSABER, d.SABER, d.FIRESABER])
@pytest.mark.parametrize("layout", sorted(LAYOUTS))
def test_layouts(engine, oracle, scheme, layout):
    with d.kem.knobs(**LAYOUTS[layout]):
        _run(engine, oracle, scheme, 101)  # partial warps of ten lanes (3), pairs (16), one lane (32)


@pytest.mark.parametrize("scheme,n", [(d.SABER, 300), (d.SABER, 301), (d.FIRESABER, 1793), (d.SABER, 4737), (d.SABER, 9472),
                                      (d.LIGHTSABER, 9473), (d.FIRESABER, 12000)])
def test_rule_edges(engine, oracle, scheme, n):
    _run(engine, oracle, scheme, n)
