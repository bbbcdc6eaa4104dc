"""The autotuner's lane sweeps force layouts that differ: at every swept size each set of knobs selects another
kernel by the launchers' rules (csrc/saber.cu, csrc/frodo.cu), and every swept product grid is one of its own."""
import pytest

from dpcrypto_b200 import autotune as at


def _saber(n, k, stage):
    warp, five = ("saber_warp_max", "saber_five_max") if stage == "saber_prologue" else (
        "saber_finish_warp_max", "saber_finish_five_max")
    return 25 if n <= k[warp] else 10 if n <= k[five] else 2 if n <= k["saber_pair_max"] else 1


def _frodo(n, k, stage):
    if stage == "frodo_prologue":  # encaps
        return 10 if n <= max(k["frodo_warp_max"], k["frodo_five_max"]) else 2 if n <= k["frodo_pair_max"] else 1
    return (25 if n <= k["frodo_ss_warp_max"] else 10 if n <= k["frodo_ss_five_max"] else
            2 if n <= k["frodo_pair_max"] else 1)


@pytest.mark.parametrize("stage", sorted(at.LAYOUTS))
def test_forced_layouts_differ(stage):
    from dpcrypto_b200 import build, kem

    build.build()
    base = {k: kem.tuning_value(k) for k in kem.RUNTIME_KNOBS + ("frodo_pair_max",)}
    layouts, _, _, form = at.LAYOUTS[stage]
    want = {"warp": 25, "five": 10, "pair": 2, "one": 1}
    saber = stage.startswith("saber")
    for n in at.SABER_SIZES if saber else at.FRODO_SIZES:
        got = {name: (_saber if saber else _frodo)(n, {**base, **kv}, stage) for name, kv in layouts.items()}
        assert got == {name: want[name] for name in layouts}, (stage, n)
    # batches of up to 1,024 run the front kernel and the stepped tail in the tensor-core form
    assert form == ("tc" if saber else "dp4a")


def test_product_grids_differ():
    assert max(at.TC_CTAS) <= 6 and len(set(at.TC_CTAS)) == len(at.TC_CTAS)  # kProductCtas in csrc/saber.cu
