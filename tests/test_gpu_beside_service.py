"""FrodoKEM batches beside an open service that holds one CTA on every SM: each call runs on what the
service leaves and returns while the service's launch is still there (a kernel that does not fit beside a
resident CTA, or that the driver has yet to load, would wait for the launch's idle exit).  In a process of
its own, so that no earlier test has loaded the kernels."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
import numpy as np, torch
import dpcrypto_b200 as d
from oracle import oracle as O

scheme, n = int(sys.argv[1]), int(sys.argv[2])
z = d.sizes(scheme)
eng, host = d.Engine(0), d.Engine(0)
kc = torch.empty((n, z["kp_coins"]), dtype=torch.uint8, device="cuda")
ec = torch.empty((n, z["enc_coins"]), dtype=torch.uint8, device="cuda")
eng.coins(n, z["kp_coins"], "beside-kp", out=kc)
eng.coins(n, z["enc_coins"], "beside-enc", out=ec)
calls = {"kp": lambda: eng.keypair(scheme, kc), "enc": lambda: eng.enc(scheme, want["kp"][0], ec),
         "dec": lambda: (eng.dec(scheme, want["enc"][0], want["kp"][1]),),
         "bad": lambda: (eng.dec(scheme, bad, want["kp"][1]),)}
want = {}
want["kp"], = [calls["kp"]()]
want["enc"], = [calls["enc"]()]
bad = want["enc"][0].clone()
bad[::2, 5] ^= 1
want["dec"], want["bad"] = calls["dec"](), calls["bad"]()
torch.cuda.synchronize()
host.set_max_ctas(torch.cuda.get_device_properties(0).multi_processor_count)
got, running = {}, {}
with d.Service(host, d.FORM_TC, idle_ms=4000) as svc:
    pk = want["kp"][0][0]
    out = [torch.empty(z[k], dtype=torch.uint8, device="cuda") for k in ("ct", "ss")]
    assert svc.submit([(scheme, 1, ec[0], pk, *out)])[0] == 1
    svc.drain()
    for name, call in calls.items():
        got[name] = call()
        torch.cuda.current_stream().synchronize()
        running[name] = bool(svc.stats()["running"]) and svc.stats()["launches"] == 1
assert all(running.values()), running
after = calls["dec"]()
for name in calls:
    for a, b in zip(got[name], want[name]):
        assert torch.equal(a, b), name
assert torch.equal(after[0], want["dec"][0]) and torch.equal(out[0], want["enc"][0][0])
idx = sorted({0, n // 2, n - 1})
h = lambda t: np.ascontiguousarray(t[idx].cpu().numpy())
pk_o, sk_o = O.keypair(scheme, h(kc), threads=8)
ct_o, ss_o = O.enc(scheme, pk_o, h(ec), threads=8)
assert (h(got["kp"][0]) == pk_o).all() and (h(got["kp"][1]) == sk_o).all()
assert (h(got["enc"][0]) == ct_o).all() and (h(got["enc"][1]) == ss_o).all() and (h(got["dec"][0]) == ss_o).all()
assert (h(got["bad"][0]) == O.dec(scheme, h(bad), sk_o, threads=8)).all()
print("ok")
"""


@pytest.mark.parametrize("scheme,n", [(0, 3), (0, 1100), (1, 5), (1, 1030)])
def test_frodo_batches_run_beside_a_service(engine, oracle, scheme, n):
    r = subprocess.run([sys.executable, "-c", CHILD, str(scheme), str(n)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout + r.stderr
