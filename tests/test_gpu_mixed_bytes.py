"""dpkem_mixed_bytes(scheme, n) is enough for a mixed batch of n requests of that scheme, whichever operations: a
context whose budget is exactly that runs it, outputs equal to the batched calls'."""
import pytest
import torch

import dpcrypto_b200 as d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op", [0, 1, 2, "all"])
@pytest.mark.parametrize("scheme,n", [(d.FRODO976, 1), (d.FRODO976, 100), (d.FRODO976AES, 25), (d.LIGHTSABER, 300),
                                      (d.FIRESABER, 7)])
def test_reservation_holds_every_operation(engine, scheme, n, op):
    z = d.sizes(scheme)
    kc = torch.empty((n, z["kp_coins"]), dtype=torch.uint8, device="cuda")
    ec = torch.empty((n, z["enc_coins"]), dtype=torch.uint8, device="cuda")
    engine.coins(n, z["kp_coins"], "mb-kp", out=kc)
    engine.coins(n, z["enc_coins"], "mb-enc", out=ec)
    pk, sk = engine.keypair(scheme, kc)
    ct, ss = engine.enc(scheme, pk, ec)
    ops = [i % 3 if op == "all" else op for i in range(n)]
    items, want, out = [], [], []
    for i, o in enumerate(ops):
        in0, in1, res = ((kc, None, (pk, sk)), (ec, pk, (ct, ss)), (ct, sk, (ss,)))[o]
        outs = [torch.zeros_like(r[i]) for r in res]
        items.append((scheme, o, in0[i], None if in1 is None else in1[i], outs[0], outs[1] if len(outs) > 1 else None))
        want += [r[i] for r in res]
        out += outs
    torch.cuda.synchronize()
    with d.Engine(0, hbm_budget=int(d.kem.load().dpkem_mixed_bytes(scheme, n))) as eng:
        eng.mixed(items, d.FORM_TC)
        eng.sync()
    torch.cuda.synchronize()
    assert all(torch.equal(o, w) for o, w in zip(out, want))
