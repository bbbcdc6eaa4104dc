"""Performance cases of the batched KEM engine, each through the public Python API.

A case is one call that a program makes: a keypair, encaps or decaps batch of one scheme on
device buffers (``path`` "batch") or on host buffers ("host"), a FrodoKEM batch under one key
with its matrix expanded once ("shared"), or a shuffled batch of all schemes and operations in
one launch ("mixed").  The outputs are bytes and have to be reproduced exactly.
"""
import math

import torch

import dpcrypto_b200 as d
from dpcrypto_b200.workloads import MixedBatch

FRODO = {"frodo976": d.FRODO976, "frodo976aes": d.FRODO976AES}
SCHEMES = {**FRODO, "lightsaber": d.LIGHTSABER, "saber": d.SABER, "firesaber": d.FIRESABER}
FORMS = {"tc": d.FORM_TC, "dp4a": d.FORM_DP4A}

# Largest batch of each path and scheme family (the sizes the benchmark and the tests run).
FRODO_MAX, SABER_MAX, HOST_MAX, MIXED_MAX, DP4A_MAX = 8192, 16384, 2048, 8192, 4096

_engine = None


def engine():
    """The one engine (device arena and streams) that a program keeps."""
    global _engine
    if _engine is None:
        _engine = d.Engine(0)
    return _engine


def listed():
    return [
        # One FrodoKEM handshake: a client encapsulates to a fresh server key.
        {"name": "frodo_enc_1", "path": "batch", "scheme": "frodo976", "op": "enc", "n": 1, "form": "tc"},
        # The handshakes that reach a server within a few milliseconds.
        {"name": "frodo_dec_32", "path": "batch", "scheme": "frodo976", "op": "dec", "n": 32, "form": "tc"},
        # Ephemeral keys made ahead of use.
        {"name": "frodo_keypair_128", "path": "batch", "scheme": "frodo976", "op": "keypair", "n": 128, "form": "tc"},
        # The batch of the reference-named entry points (768), on pinned host buffers.
        {"name": "frodo_enc_768_host", "path": "host", "scheme": "frodo976", "op": "enc", "n": 768, "form": "tc"},
        # The headline batch.
        {"name": "frodo_enc_8192", "path": "batch", "scheme": "frodo976", "op": "enc", "n": 8192, "form": "tc"},
        # The AES variant at a ragged ordinary size.
        {"name": "frodoaes_dec_333", "path": "batch", "scheme": "frodo976aes", "op": "dec", "n": 333, "form": "tc"},
        # A server that decapsulates under its own long-lived key.
        {"name": "frodo_shared_dec_4096", "path": "shared", "scheme": "frodo976", "op": "dec", "n": 4096, "form": "tc"},
        # One Saber handshake: the smallest call.
        {"name": "saber_enc_1", "path": "batch", "scheme": "saber", "op": "enc", "n": 1, "form": "tc"},
        # The Saber batch of the benchmark.
        {"name": "saber_dec_4096", "path": "batch", "scheme": "saber", "op": "dec", "n": 4096, "form": "tc"},
        # The dot-product form, which the reference calls mode 0, at an odd ordinary size.
        {"name": "firesaber_enc_1501_dp", "path": "batch", "scheme": "firesaber", "op": "enc", "n": 1501, "form": "dp4a"},
        # A large stock of ephemeral keys of the lightest scheme.
        {"name": "lightsaber_keypair_16384", "path": "batch", "scheme": "lightsaber", "op": "keypair", "n": 16384,
         "form": "tc"},
        # A gateway's queue: four schemes, three operations, one launch.
        {"name": "mixed_4096", "path": "mixed", "scheme": "all", "op": "all", "n": 4096, "form": "tc"},
    ]


def _log_uniform(rng, hi):
    return max(1, min(hi, int(round(math.exp(rng.uniform(0.0, math.log(hi)))))))


def draw(rng):
    path = rng.choice(["batch"] * 8 + ["host", "shared", "mixed"])
    if path == "mixed":
        return {"path": path, "scheme": "all", "op": "all", "n": max(64, _log_uniform(rng, MIXED_MAX)), "form": "tc"}
    if path == "shared":
        return {"path": path, "scheme": rng.choice(sorted(FRODO)), "op": rng.choice(["enc", "dec"]),
                "n": _log_uniform(rng, FRODO_MAX), "form": "tc"}
    scheme = rng.choice(["frodo976", "frodo976", "frodo976aes", "lightsaber", "saber", "firesaber"])
    form = rng.choice(["tc"] * 5 + ["dp4a"])
    hi = HOST_MAX if path == "host" else FRODO_MAX if scheme in FRODO else SABER_MAX
    if form == "dp4a":
        hi = min(hi, DP4A_MAX)
    return {"path": path, "scheme": scheme, "op": rng.choice(["keypair", "enc", "dec"]), "n": _log_uniform(rng, hi),
            "form": form}


def _random_bytes(n, length, gen):
    return torch.randint(0, 256, (n, length), dtype=torch.uint8, device="cuda", generator=gen)


def _tamper(ct):
    """Every 64th ciphertext arrives with a flipped bit (implicit rejection)."""
    idx = torch.arange(0, ct.shape[0], 64, device=ct.device)
    ct[idx, (idx * 7919) % ct.shape[1]] ^= 1
    return ct


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def prepare(case, seed):
    eng, form, n, op = engine(), FORMS[case["form"]], case["n"], case["op"]
    if case["path"] == "mixed":
        # the queue's order belongs to the case; keys, coins and ciphertexts come from the seed
        mb = MixedBatch(eng, n, seed=n, first=1000003 * seed)
        return {"case": case, "eng": eng, "form": form, "batch": mb, "table": eng.requests(mb.items)}
    scheme = SCHEMES[case["scheme"]]
    z = d.sizes(scheme)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    st = {"case": case, "eng": eng, "form": form, "scheme": scheme}
    shared = case["path"] == "shared"
    kc = _random_bytes(1 if shared else n, z["kp_coins"], gen)
    ec = _random_bytes(n, z["enc_coins"], gen)
    if op == "keypair":
        args, outs = (kc,), ("pk", "sk")
    else:
        pk, sk = eng.keypair(scheme, kc)
        if shared:
            pk, sk = pk[0].contiguous(), sk[0].contiguous()
            st["amat"] = eng.expand_a(scheme, pk)
        if op == "enc":
            args, outs = (pk, ec), ("ct", "ss")
        else:
            ct = (eng.enc_shared(scheme, pk, ec, amat=st["amat"]) if shared else eng.enc(scheme, pk, ec))[0]
            args, outs = (_tamper(ct), sk), ("ss",)
    if case["path"] == "host":
        torch.cuda.synchronize()
        out = [torch.empty((n, z[k]), dtype=torch.uint8, pin_memory=True).numpy() for k in outs]
        st["out"] = out[0] if len(out) == 1 else tuple(out)
        args = tuple(_pinned(a) for a in args)
    st["args"] = args
    return st


def run(state):
    case, eng, form = state["case"], state["eng"], state["form"]
    if case["path"] == "mixed":
        eng.mixed(state["table"], form)
        return state["batch"].outputs
    if case["path"] == "shared":
        call = eng.enc_shared if case["op"] == "enc" else eng.dec_shared
        return call(state["scheme"], *state["args"], form=form, amat=state["amat"])
    return getattr(eng, case["op"])(state["scheme"], *state["args"], form=form, out=state.get("out"))


# Integer operations of one Keccak-f[1600] (180 LOP3 / SHF per round) and of one AES-128 block
# (10 rounds x 4 columns x 4 byte lookups, each a byte extract, a lookup and an XOR).
_KECCAK, _AES = 4320, 480


def _ops(scheme, op, shared=False):
    """Integer operations of one instance: permutations or AES blocks, and multiply-adds."""
    if scheme in FRODO:
        macs = 8 * 976 * 976 + (0 if op == "keypair" else 64 * 976) + (64 * 976 if op == "dec" else 0)
        rows = 0 if shared else 976 * (12 * _KECCAK if scheme == "frodo976" else 122 * _AES)
        chain = {"keypair": 1 + 230 + 115, "enc": (0 if shared else 115) + 1 + 231 + 116, "dec": 1 + 231 + 116}[op]
        return 2 * macs + rows + chain * _KECCAK
    lv = {"lightsaber": 2, "saber": 3, "firesaber": 4}[scheme]
    mu = {2: 10, 3: 8, 4: 6}[lv]
    blocks = lambda nbytes, rate: nbytes // rate + 1  # noqa: E731
    z = d.sizes(SCHEMES[scheme])
    polys = lv * lv + {"keypair": 0, "enc": lv, "dec": 2 * lv}[op]
    xof = -(-lv * lv * 416 // 168) + -(-lv * mu * 32 // 168)
    chain = {"keypair": 1 + blocks(z["pk"], 136), "enc": 3 + blocks(z["pk"], 136) + blocks(z["ct"], 136),
             "dec": 2 + blocks(z["ct"], 136)}[op]
    return 2 * polys * 256 * 256 + (xof + chain) * _KECCAK


def _bytes(scheme, op):
    z = d.sizes(SCHEMES[scheme])
    return sum(z[k] for k in {"keypair": ("kp_coins", "pk", "sk"), "enc": ("enc_coins", "pk", "ct", "ss"),
                              "dec": ("ct", "sk", "ss")}[op])


def work(case):
    n = case["n"]
    if case["path"] == "mixed":
        kinds = [(s, o) for s in ("frodo976", "lightsaber", "saber", "firesaber") for o in ("keypair", "enc", "dec")]
        return {"bytes": n * sum(_bytes(*k) for k in kinds) / len(kinds),
                "flops": n * sum(_ops(*k) for k in kinds) / len(kinds)}
    scheme, op = case["scheme"], case["op"]
    if case["path"] == "shared":
        z = d.sizes(SCHEMES[scheme])
        each = z["ct"] + z["ss"] + (z["enc_coins"] if op == "enc" else 0)
        return {"bytes": n * each + z["pk" if op == "enc" else "sk"] + 976 * 976 * 2, "flops": n * _ops(scheme, op, True)}
    return {"bytes": n * _bytes(scheme, op), "flops": n * _ops(scheme, op)}


def exact(case, seed):
    """Every output is bytes (keys, ciphertexts, hashes), compared as they are."""
    return None
