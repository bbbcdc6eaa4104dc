"""FrodoKEM prologues outside the tensor-core batches with a key per instance (one key, dot-product forms) on
both sides of the sizes at which their layout changes: every instance against the calls with a key per
instance, a sample against the CPU oracle, tampered ciphertexts among them."""
import os

import numpy as np
import pytest
import torch

import dpcrypto_b200 as d

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 8


def _keys(engine, scheme, n):
    kc = torch.empty((1, 64), dtype=torch.uint8, device="cuda")
    ec = torch.empty((n, 24), dtype=torch.uint8, device="cuda")
    engine.coins(1, 64, "prol-kp", out=kc)
    engine.coins(n, 24, "prol-enc", out=ec)
    pk, sk = engine.keypair(scheme, kc)
    return pk[0].contiguous(), sk[0].contiguous(), ec


def _tamper(ct):
    bad = ct.clone()
    n = ct.shape[0]
    i = torch.arange(0, n, 3, device="cuda")
    bad[i, (i * 7919) % ct.shape[1]] ^= 16
    return bad


# chains of encaps end at 6,144, of decaps at 5,600, pairs at 9,472
@pytest.mark.parametrize("n", [4096, 4097, 5600, 5601, 6144, 6145, 9472, 9473])
def test_one_key(engine, oracle, n):
    pk, sk, ec = _keys(engine, d.FRODO976, n)
    amat = engine.expand_a(d.FRODO976, pk)
    ct, ss = engine.enc_shared(d.FRODO976, pk, ec, amat=amat)
    many_pk = pk.expand(n, -1).contiguous()
    ct2, ss2 = engine.enc(d.FRODO976, many_pk, ec)
    assert torch.equal(ct, ct2) and torch.equal(ss, ss2)
    del many_pk, ct2
    bad = _tamper(ct)
    got = engine.dec_shared(d.FRODO976, bad, sk, amat=amat)
    many_sk = sk.expand(n, -1).contiguous()
    assert torch.equal(got, engine.dec(d.FRODO976, bad, many_sk))
    same = (got == ss).all(dim=1)
    assert not same[::3].any() and same[1::3].all() and same[2::3].all()
    idx = sorted({0, 1, n // 2, n - 1})
    h = lambda t: np.ascontiguousarray(t[idx].cpu().numpy())  # noqa: E731
    ct_o, ss_o = oracle.enc(0, np.repeat(pk.cpu().numpy()[None], len(idx), 0), h(ec), threads=THREADS)
    assert (h(ct) == ct_o).all() and (h(ss) == ss_o).all()
    assert (h(got) == oracle.dec(0, h(bad), np.repeat(sk.cpu().numpy()[None], len(idx), 0), threads=THREADS)).all()


@pytest.mark.parametrize("form,n", [(d.FORM_DP4A, 683), (d.FORM_DP4A, 684), (d.FORM_INT32, 1024), (d.FORM_DP4A, 1025)])
def test_small_chain_limit(engine, oracle, form, n):
    """Chains up to 1,024, decaps likewise (the limit of a program that sets no knobs before the defaults
    were raised)."""
    with d.kem.knobs(frodo_warp_max=1024, frodo_five_max=0):
        pk, sk, ec = _keys(engine, d.FRODO976, n)
        ct, ss = engine.enc_shared(d.FRODO976, pk, ec, form)
        bad = _tamper(ct)
        got = engine.dec_shared(d.FRODO976, bad, sk, form)
        same = (got == ss).all(dim=1)
        assert not same[::3].any() and same[1::3].all() and same[2::3].all()
        idx = [0, 1, n - 1]
        h = lambda t: np.ascontiguousarray(t[idx].cpu().numpy())  # noqa: E731
        assert (h(got) == oracle.dec(0, h(bad), np.repeat(sk.cpu().numpy()[None], 3, 0), threads=THREADS)).all()


BIG = 1 << 30
PROLOGUES = {"chains": dict(frodo_warp_max=0, frodo_five_max=BIG),
             "pair": dict(frodo_warp_max=0, frodo_five_max=0, frodo_pair_max=BIG),
             "one": dict(frodo_warp_max=0, frodo_five_max=0, frodo_pair_max=0)}
HASHES = {"warp": dict(frodo_ss_warp_max=BIG), "ten": dict(frodo_ss_warp_max=0, frodo_ss_five_max=BIG),
          "pair": dict(frodo_ss_warp_max=0, frodo_ss_five_max=0, frodo_pair_max=BIG),
          "one": dict(frodo_ss_warp_max=0, frodo_ss_five_max=0, frodo_pair_max=0)}


# n = 50 and 67 leave partial groups of three, sixteen and thirty-two; the pair limit is common to both stages
@pytest.mark.parametrize("n", [1, 50, 67])
@pytest.mark.parametrize("scheme,form", [(d.FRODO976, d.FORM_DP4A), (d.FRODO976AES, d.FORM_INT32)])
@pytest.mark.parametrize("prologue,hash_", [("chains", "warp"), ("chains", "ten"), ("chains", "pair"), ("chains", "one"),
                                            ("pair", "pair"), ("pair", "warp"), ("one", "one"), ("one", "ten")])
def test_layouts(engine, oracle, scheme, form, prologue, hash_, n):
    kc = torch.empty((n, 64), dtype=torch.uint8, device="cuda")
    ec = torch.empty((n, 24), dtype=torch.uint8, device="cuda")
    engine.coins(n, 64, "prol-kp", first=n, out=kc)
    engine.coins(n, 24, "prol-enc", first=n, out=ec)
    h = lambda t: t.cpu().numpy()  # noqa: E731
    pk_o, sk_o = oracle.keypair(scheme, h(kc), threads=THREADS)
    ct_o, ss_o = oracle.enc(scheme, pk_o, h(ec), threads=THREADS)
    bad = torch.from_numpy(ct_o).cuda()
    bad[::2, 15743] ^= 128
    rej_o = oracle.dec(scheme, h(bad), sk_o, threads=THREADS)
    with d.kem.knobs(**{**HASHES[hash_], **PROLOGUES[prologue]}):
        pk, sk = engine.keypair(scheme, kc, form)
        ct, ss = engine.enc(scheme, pk, ec, form)
        rej = engine.dec(scheme, bad, sk, form)
        tc = engine.dec(scheme, bad, sk, d.FORM_TC)  # its final hash
    assert (h(pk) == pk_o).all() and (h(sk) == sk_o).all()
    assert (h(ct) == ct_o).all() and (h(ss) == ss_o).all()
    assert (h(rej) == rej_o).all() and (h(tc) == rej_o).all()
