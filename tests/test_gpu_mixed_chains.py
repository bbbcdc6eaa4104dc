"""Planned mixed batches on both sides of the rule for FrodoKEM's chain tasks: a group of 1,152 requests and of
one more, in a mix that is more than half Saber and in one that is not.  Every output against the batched calls, a
sample against the CPU oracle."""
import numpy as np
import pytest
import torch

import dpcrypto_b200 as d

pytestmark = pytest.mark.gpu


def _group(engine, scheme, op, n, items, expect):
    z = d.sizes(scheme)
    kc = torch.empty((n, z["kp_coins"]), dtype=torch.uint8, device="cuda")
    ec = torch.empty((n, z["enc_coins"]), dtype=torch.uint8, device="cuda")
    engine.coins(n, z["kp_coins"], "mch-kp", first=op * 10000, out=kc)
    engine.coins(n, z["enc_coins"], "mch-enc", first=op * 10000, out=ec)
    pk, sk = engine.keypair(scheme, kc, d.FORM_DP4A)
    ct, ss = engine.enc(scheme, pk, ec, d.FORM_DP4A)
    if op == 2:
        ct = ct.clone()
        ct[::2, 3] ^= 1
        ss = engine.dec(scheme, ct, sk, d.FORM_DP4A)
    in0, in1, want = ((kc, None, (pk, sk)), (ec, pk, (ct, ss)), (ct, sk, (ss,)))[op]
    out = [torch.zeros_like(w) for w in want]
    items += [(scheme, op, in0[i], None if in1 is None else in1[i], out[0][i], out[1][i] if len(out) > 1 else None)
              for i in range(n)]
    expect += list(zip(out, want))


@pytest.mark.parametrize("op", [0, 1, 2])
@pytest.mark.parametrize("frodo,saber", [(1152, 1200), (1153, 1200), (1153, 1100)])
@pytest.mark.parametrize("scheme", [d.FRODO976])
def test_chain_group_limit(engine, oracle_check_items, scheme, op, frodo, saber):
    items, expect = [], []
    _group(engine, scheme, op, frodo, items, expect)
    _group(engine, d.LIGHTSABER, (op + 1) % 3, saber, items, expect)
    order = np.random.default_rng(op).permutation(len(items))
    items = [items[k] for k in order]
    torch.cuda.synchronize()
    engine.mixed(items, d.FORM_TC)
    engine.sync()
    torch.cuda.synchronize()
    for got, want in expect:
        assert torch.equal(got, want)
    assert oracle_check_items(items, 997, offset=3) >= 2


@pytest.mark.parametrize("scheme,n", [(d.FRODO976AES, 37), (d.FRODO976, 13), (d.FRODO976, 1)])
def test_chain_tasks_with_partial_groups(engine, oracle_check_items, scheme, n):
    """Tasks of twelve (decaps six, hashes twenty-four) with a remainder, all three operations in one launch."""
    items, expect = [], []
    for op in range(3):
        _group(engine, scheme, op, n + op, items, expect)
    torch.cuda.synchronize()
    engine.mixed(items, d.FORM_TC)
    engine.sync()
    torch.cuda.synchronize()
    for got, want in expect:
        assert torch.equal(got, want)
    assert oracle_check_items(items, 7) >= 1
