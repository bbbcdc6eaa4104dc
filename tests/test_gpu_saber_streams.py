"""Saber decaps whose GenMatrix runs on a second stream: from the chunks of a host-buffer batch, and from two
contexts in two threads on streams of their own.  Against the INT32 form and the CPU oracle."""
import threading

import numpy as np
import pytest
import torch

import dpcrypto_b200 as d

pytestmark = pytest.mark.gpu


def _case(engine, scheme, n, first=0):
    z = d.sizes(scheme)
    kc = torch.empty((n, z["kp_coins"]), dtype=torch.uint8, device="cuda")
    ec = torch.empty((n, z["enc_coins"]), dtype=torch.uint8, device="cuda")
    engine.coins(n, z["kp_coins"], "str-kp", first=first, out=kc)
    engine.coins(n, z["enc_coins"], "str-enc", first=first, out=ec)
    pk, sk = engine.keypair(scheme, kc, d.FORM_INT32)
    ct, _ = engine.enc(scheme, pk, ec, d.FORM_INT32)
    ct[::3, 7] ^= 2
    return ct, sk, engine.dec(scheme, ct, sk, d.FORM_INT32)


# chunks of 256, of 300, and of 128 / 512 / 128 (up to 300 instances take the second stream)
@pytest.mark.parametrize("n", [512, 600, 768])
@pytest.mark.parametrize("scheme,form", [(d.SABER, d.FORM_TC), (d.FIRESABER, d.FORM_TC), (d.SABER, d.FORM_DP4A)])
def test_host_chunks(engine, oracle, scheme, form, n):
    ct, sk, ss = _case(engine, scheme, n)
    h_ct, h_sk = (t.cpu().pin_memory().numpy() for t in (ct, sk))
    for _ in range(3):
        got = engine.dec(scheme, h_ct, h_sk, form)
        assert (got == ss.cpu().numpy()).all()
    idx = [0, 1, n - 1]
    assert (got[idx] == oracle.dec(scheme, np.ascontiguousarray(h_ct[idx]), np.ascontiguousarray(h_sk[idx]), threads=3)).all()


@pytest.mark.parametrize("sizes", [(300, 257), (12000, 300)])
def test_two_contexts_at_once(engine, sizes):
    cases = [_case(engine, s, n, first=n) for s, n in zip((d.SABER, d.FIRESABER), sizes)]
    torch.cuda.synchronize()
    bad = []

    def work(scheme, case):
        ct, sk, ss = case
        with d.Engine(0) as eng, torch.cuda.stream(torch.cuda.Stream()):
            outs = [torch.zeros_like(ss) for _ in range(20)]
            torch.cuda.current_stream().synchronize()
            for o in outs:
                eng.dec(scheme, ct, sk, d.FORM_TC, out=o)
            torch.cuda.current_stream().synchronize()
            bad.extend(1 for o in outs if not torch.equal(o, ss))
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(s, c)) for s, c in zip((d.SABER, d.FIRESABER), cases)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
