"""A context's arena and FrodoKEM's operand tiles: calls captured on a reserved context, captured calls
replayed after the arena has grown, reserved contexts that allocate nothing.  Against the session's engine and
the CPU oracle."""
import numpy as np
import pytest
import torch

import dpcrypto_b200 as d

pytestmark = pytest.mark.gpu


def _inputs(engine, n):
    kc = torch.empty((n, 64), dtype=torch.uint8, device="cuda")
    ec = torch.empty((n, 24), dtype=torch.uint8, device="cuda")
    engine.coins(n, 64, "arena-kp", out=kc)
    engine.coins(n, 24, "arena-enc", out=ec)
    pk, sk = engine.keypair(d.FRODO976, kc)
    ct, ss = engine.enc(d.FRODO976, pk, ec)
    bad = ct.clone()
    bad[::2, 11] ^= 1
    return {"keypair": ((kc,), (pk, sk)), "enc": ((pk, ec), (ct, ss)),
            "dec": ((bad, sk), (engine.dec(d.FRODO976, bad, sk, d.FORM_DP4A),))}


# 64 MB hold the tiles of 29 instances: all of 20, none or some of 60
@pytest.mark.parametrize("n", [3, 20, 60])
@pytest.mark.parametrize("op", ["keypair", "enc", "dec"])
def test_captured_on_a_reserved_context(engine, op, n):
    args, want = _inputs(engine, n)[op]
    static = [a.clone() for a in args]
    out = [torch.zeros_like(w) for w in want]
    torch.cuda.synchronize()
    with d.Engine(0) as eng:
        eng.reserve(64 << 20)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            getattr(eng, op)(d.FRODO976, *static, out=tuple(out) if len(out) > 1 else out[0])
        for _ in range(2):
            for o in out:
                o.zero_()
            g.replay()
            torch.cuda.synchronize()
            assert all(torch.equal(o, w) for o, w in zip(out, want))
        # the arena grows, and what it was gets other contents if it has gone back to the device
        eng.reserve(256 << 20)
        fill = torch.full((300 << 20,), 0xA5, dtype=torch.uint8, device="cuda")
        for o in out:
            o.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(o, w) for o, w in zip(out, want))
        assert bool((fill == 0xA5).all())
        del g


def test_capture_needs_a_reserved_arena(engine):
    """Without one the call is refused, and the context works on."""
    args, want = _inputs(engine, 4)["enc"]
    torch.cuda.synchronize()
    with d.Engine(0) as eng:
        g = torch.cuda.CUDAGraph()
        out = tuple(torch.zeros_like(w) for w in want)
        with torch.cuda.graph(g):
            with pytest.raises(d.DpkemError):
                eng.enc(d.FRODO976, *args, out=out)
        got = eng.enc(d.FRODO976, *args)
        assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_reserved_context_allocates_nothing(engine, oracle):
    n = 300
    cases = _inputs(engine, n)
    for _ in range(2):  # the first pass loads the kernels
        with d.Engine(0) as eng:
            eng.reserve(128 << 20)
            torch.cuda.synchronize()
            free = torch.cuda.mem_get_info()[0]
            for op, (args, want) in cases.items():
                for m in (1, 30, n):
                    part = [a[:m] for a in args]
                    out = tuple(torch.empty_like(w[:m]) for w in want)
                    getattr(eng, op)(d.FRODO976, *part, out=out if len(out) > 1 else out[0])
                    eng.sync()
                    assert all(torch.equal(o, w[:m]) for o, w in zip(out, want)), (op, m)
            torch.cuda.synchronize()
            after = torch.cuda.mem_get_info()[0]
    assert free - after < 32 << 20  # the outputs' pool at most; 300 instances' tiles are 649 MB
    idx = [0, n - 1]
    h = lambda t: np.ascontiguousarray(t[idx].cpu().numpy())  # noqa: E731
    (pk, ec), (ct, ss) = cases["enc"]
    ct_o, ss_o = oracle.enc(0, h(pk), h(ec), threads=2)
    assert (h(ct) == ct_o).all() and (h(ss) == ss_o).all()
