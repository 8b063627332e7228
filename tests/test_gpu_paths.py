"""Launch variants of the solver and marker kernels at the sizes and boundary rows where they could
differ from the general path."""
import numpy as np
import pytest

import cases
import oracle as O
from conftest import golden
from i3elvis_b200 import abi, config, lib, model

pytestmark = pytest.mark.gpu


def _random_box(shape, multinum, seed):
    """A free-slip box of any shape with lognormal nodal viscosities and random densities."""
    spec = model.ModelSpec(shape=shape, size=tuple(1e3 * (n - 1) for n in shape), multinum=multinum)
    one = np.full(1, 500.0, np.float32)
    prn = model.make_prn(spec, {model.MATRIX: model.Rock()}, np.full(1, model.MATRIX, np.int8), (one, one, one))
    rng = np.random.default_rng(seed)
    n = prn.nodenum
    for f in ("nu", "nxx", "nxy", "nxz", "nyz"):
        prn.nodes[f] = (1e21 * np.exp(rng.normal(0, 1.5, n))).astype(np.float32)
    prn.nodes["ro"] = rng.uniform(3200, 3400, n).astype(np.float32)
    mode = config.Mode(multinum=multinum, multicyc=1, multinnn=((2,) * multinum + (0,), (2,) * multinum + (3,)), p0koef=0.71, p1koef=0.5,
                       nubeg=1e18, nuend=1e25, files=[config.OutFile("o.prn", nubeg=1e18, nuend=1e25, p0koef=0.71, p1koef=0.5,
                                                                     multinum=multinum, multinum2=multinum)])
    return prn, mode


def _vcycles_match(p, mode):
    par, fp = abi.make_params(mode), abi.make_file_params(mode.files[0])
    g = lib.Context(abi.ModelBuffers(p), par, fp)
    o = O.Oracle(abi.ModelBuffers(p), par, fp)
    g.call("i3g_stokes_setup")
    o.call("orc_stokes_setup")
    g.call("i3g_stokes_vcycles", 2)
    o.call("orc_stokes_vcycles_mc", 2)
    for l, n in enumerate(cases.level_sizes(p, mode.multinum)):
        a, b = g.get(abi.A_SOL, l, 4 * n), o.get(abi.A_SOL, l, 4 * n)
        assert np.all(np.isfinite(b)) and np.any(b != 0)
        assert np.array_equal(a, b), l
    g.close()


# levels relaxed with the early prologue (default), and all without it
PROLOGUE = ["400000", "0"]


@pytest.mark.parametrize("pro", PROLOGUE)
@pytest.mark.parametrize("factor", [-1.0, 0.0, 0.5])
def test_vcycles_bit_exact_for_wall_factors(factor, pro, monkeypatch):
    """Boundary rows x = k x_partner with k = -1 and 0 take the packed form, k = 0.5 the general one;
    chains along edges and corners multiply the factors.  Both equal the oracle bit for bit."""
    monkeypatch.setenv("I3G_PRO_NODES", pro)
    p, mode, _ = golden("sphere17")
    b = p.bond
    vel = (b["row"] < 4 * sum(cases.level_sizes(p, mode.multinum))) & (b["row"] % 4 != 0) & (b["partner1"] > 0)
    assert vel.sum() > 1000
    b["k"][vel] = factor
    _vcycles_match(p, mode)


@pytest.mark.parametrize("pro", PROLOGUE)
@pytest.mark.parametrize("shape,multinum", [((9, 9, 9), 0), ((13, 19, 15), 2), ((21, 13, 17), 1), ((12, 10, 14), 0)])
def test_vcycles_bit_exact_on_boxes(shape, multinum, pro, monkeypatch):
    monkeypatch.setenv("I3G_PRO_NODES", pro)
    _vcycles_match(*_random_box(shape, multinum, seed=sum(shape)))
