"""Launch variants of the solver and marker kernels at the sizes and boundary rows where they could
differ from the general path."""
import numpy as np
import pytest

import cases
import oracle as O
import unet_ref as U
from conftest import golden
from i3elvis_b200 import abi, config, lib, model, warmstart
from i3elvis_b200.prn import ROCK_FIELDS
from test_oracle_markers import marker_setup

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


def test_vcycles_of_a_level_beyond_the_row_indexed_table(monkeypatch):
    """Level 1 has 456,225 nodes: its packed boundary entries are found through the writer list, not the
    table indexed by the row.  Bit for bit the same as one launch per boundary pass."""
    sols = []
    for fuse in ("1", "0"):
        monkeypatch.setenv("I3G_FUSE", fuse)
        p, mode = _random_box((149, 145, 153), 1, seed=7)
        assert cases.level_sizes(p, 1)[1] > 400000
        g = lib.Context(abi.ModelBuffers(p), abi.make_params(mode), abi.make_file_params(mode.files[0]))
        g.call("i3g_stokes_setup")
        g.call("i3g_stokes_vcycles", 1)
        sols.append([g.get(abi.A_SOL, l, 4 * n) for l, n in enumerate(cases.level_sizes(p, 1))])
        g.close()
    for a, b in zip(*sols):
        assert np.all(np.isfinite(a)) and np.any(a != 0)
        assert np.array_equal(a, b)


@pytest.mark.parametrize("pro", ["1100000", "0"])
def test_vcycles_with_and_without_prologue_beyond_the_row_indexed_table(pro, monkeypatch):
    """The level of 456,225 nodes again, its packed entries read before and after the wait for the
    predecessor: the solution of one launch per boundary pass bit for bit."""
    sols = []
    for fuse in ("1", "0"):
        monkeypatch.setenv("I3G_FUSE", fuse)
        monkeypatch.setenv("I3G_PRO_NODES", pro)
        p, mode = _random_box((149, 145, 153), 1, seed=8)
        g = lib.Context(abi.ModelBuffers(p), abi.make_params(mode), abi.make_file_params(mode.files[0]))
        g.call("i3g_stokes_setup")
        g.call("i3g_stokes_vcycles", 1)
        sols.append([g.get(abi.A_SOL, l, 4 * n) for l, n in enumerate(cases.level_sizes(p, 1))])
        g.close()
    for a, b in zip(*sols):
        assert np.all(np.isfinite(a)) and np.any(a != 0)
        assert np.array_equal(a, b)


def _cloud(seed=5):
    """Reference fields of the 13^3 case with markers of every rock moved to uneven places: empty cells,
    cells of a few markers and cells of several hundred (more than a warp stages at once)."""
    p, mode, fx, buf = marker_setup("sphere13")
    rng = np.random.default_rng(seed)
    n = buf.f32["markx"].size
    L = 1e5
    for f in ("markx", "marky", "markz"):
        a = rng.uniform(0.001 * L, 0.999 * L, n)
        a[: n // 2] = rng.uniform(0.30 * L, 0.42 * L, n // 2)
        buf.f32[f][:] = a
    buf.f32["markk"][:] = rng.uniform(300, 1500, n)
    buf.f32["markv"][:] = 1e21 * np.exp(rng.normal(0, 2, n))
    return p, mode, fx, buf


NODE_SUMS = ("ro", "nu", "nxx", "nxy", "nxz", "nyz", "tk", "cp", "kt", "et", "ht", "rr")


def _nodes_match(mode, dt, edit, exact, **fields):
    bufs = []
    for side in range(2):
        _, _, _, buf = _cloud()
        edit(buf)
        par, fp = abi.make_params(mode, marker_exact=exact), abi.make_file_params(mode.files[0])
        for k, v in fields.items():
            setattr(par, k, v)
        c = lib.Context(buf, par, fp) if side == 0 else O.Oracle(buf, par, fp)
        if side == 0:
            c.markers_to_nodes(dt)
        else:
            c.call("orc_markers_to_nodes", dt)
        c.download(abi.SYNC_ALL)
        c.close()
        bufs.append(buf)
    for f in NODE_SUMS:   # FP64 sums in another order, stored as FP32
        np.testing.assert_allclose(bufs[0].f32[f], bufs[1].f32[f], rtol=3e-7, atol=0, err_msg=f)
    np.testing.assert_allclose(bufs[0].f32["markv"], bufs[1].f32["markv"], rtol=2e-7)


@pytest.mark.parametrize("exact", [0, 1])
@pytest.mark.parametrize("viscmod,nukoef", [(0, 0.0), (1, 0.0), (2, 0.3)])
def test_node_sums_of_uneven_cells(viscmod, nukoef, exact):
    """Marker -> node sums over cells of 0 to several hundred markers, the three viscosity averages
    and the nukoef gate, against the oracle."""
    _, mode, _, _ = _cloud()
    _nodes_match(mode, 1e10, lambda buf: None, exact, viscmod=viscmod, nukoef=nukoef)


@pytest.mark.parametrize("exact", [0, 1])
def test_node_sums_with_markers_without_viscosity(exact):
    """A marker whose viscosity is still 0 in a time step gets one from the rheology, as in the
    initial passes; the others' sums stay the same."""
    _, mode, _, _ = _cloud()

    def edit(buf):
        buf.f32["markv"][[7, 300, 9000]] = 0.0
    _nodes_match(mode, 1e10, edit, exact)


@pytest.mark.parametrize("exact", [0, 1])
@pytest.mark.parametrize("field,value", [("markrr", np.inf), ("markrr", -np.inf), ("markrr", np.nan), ("markv", np.inf)])
def test_node_sums_with_a_marker_that_is_not_finite(field, value, exact):
    """A property that is not finite reaches the nodes its marker weighs on and no other: 0 x inf is NaN in a
    matrix product.  Markers in crowded, sparse and otherwise empty cells, beside nodes without markers, which
    keep what they had."""
    _, mode, _, base = _cloud()
    x, y, z = (base.f32[f] for f in ("markx", "marky", "markz"))
    cell = (z / 8334).astype(int) * 144 + (x / 8334).astype(int) * 12 + (y / 8334).astype(int)
    count = np.bincount(cell, minlength=1728)[cell]
    at = [int(np.flatnonzero(count == count.max())[0])] + [int(i) for i in np.flatnonzero(count <= 2)[:3]]
    empty = (x > 6e4) & (y > 6e4)   # leave this corner to one marker
    keep = int(np.flatnonzero(empty)[0])

    def edit(buf):
        for f in ("markx", "marky"):
            a = buf.f32[f][empty]
            buf.f32[f][empty] = a - 5e4
        for f, v in (("markx", 8.1e4), ("marky", 8.3e4), ("markz", 5.2e4)):
            buf.f32[f][keep] = v
        buf.f32[field][at + [keep]] = value
        for f in NODE_SUMS:
            if f not in ("nu", "tk"):
                buf.f32[f][:] = 7.0
    _nodes_match(mode, 1e10, edit, exact)


def test_two_contexts_of_different_sizes():
    """A smaller model created while a larger one is alive leaves the larger one's marker and heat kernels the
    shared memory they need: the results are those of the model alone."""
    def run(other):
        p, mode, fx, buf = marker_setup("dp17")
        g = lib.Context(buf, abi.make_params(mode), abi.make_file_params(mode.files[0]))
        if other:
            p2, mode2, _, buf2 = marker_setup("sphere13")
            h = lib.Context(buf2, abi.make_params(mode2), abi.make_file_params(mode2.files[0]))
        dt = float(fx["fld_dt"][0])
        g.heat(0, dt)
        g.move_markers(dt)
        g.markers_to_nodes(dt)
        if other:
            h.markers_to_nodes(0.0)
            h.close()
        g.markers_to_nodes(0.0)
        g.download(abi.SYNC_ALL)
        g.close()
        return buf
    alone, beside = run(False), run(True)
    for f in NODE_SUMS + ("markx", "markk", "markv"):
        assert np.array_equal(alone.f32[f], beside.f32[f]), f


def test_bytes_of_a_marker_move_count_the_fields_it_reads():
    """Strain rates and stresses (12 FP32 fields) count only where a rock of the model reads their invariants."""
    per_node = {}
    for name in ("sphere13", "dp17"):
        p, mode, _, buf = marker_setup(name)
        g = lib.Context(buf, abi.make_params(mode), abi.make_file_params(mode.files[0]))
        per_node[name] = (g.time_kernel(5, 1)[1] - 45.0 * buf.f32["markx"].size) / p.nodenum
        g.close()
    assert per_node == {"sphere13": 20.0, "dp17": 68.0}


def test_closed_contexts_give_their_memory_back():
    """The tables of a level share allocations that belong to the level: thirty models created and closed leave
    the device with the memory it had after the first (the driver hands out 2 MB at a time)."""
    import torch
    p, mode, _, buf = marker_setup("sphere13")
    par, fp = abi.make_params(mode, precision=1, krylov=8, stokes_rtol=1e-4), abi.make_file_params(mode.files[0])
    free = []
    for k in range(31):
        g = lib.Context(buf, par, fp)
        if k % 10 == 0:
            g.stokes(0, 1e30)
        g.close()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[-1] <= 4 << 20, [free[0] - f for f in free]


def test_partial_download_after_a_sort():
    """A download that names a few marker arrays returns those in the original order, and fields that
    the sort does not move stay with their markers."""
    p, mode, fx, buf = marker_setup("sphere13")
    n = buf.f32["markx"].size
    rng = np.random.default_rng(9)
    for f in ("markw", "markd", "markex", "markft", "markrn"):
        buf.f32[f][:] = rng.uniform(0, 1, n)
    keep = {f: buf.f32[f].copy() for f in ("markw", "markd", "markex", "markft", "markrn")}
    g = lib.Context(buf, abi.make_params(mode), abi.make_file_params(mode.files[0]))
    g.move_markers(float(fx["fld_dt"][0]))
    g.markers_to_nodes(1e10)
    g.download(abi.SYNC_MARKERS)
    whole = {f: buf.f32[f].copy() for f in abi.MARK_F32}
    for f, v in keep.items():
        assert np.array_equal(whole[f], v), f
    part = abi.Model.from_buffer_copy(buf.model)
    got = np.zeros(n, np.float32)
    for f in abi.MARK_F32:
        setattr(part, f, got.ctypes.data_as(abi.c_f32p) if f == "marky" else abi.c_f32p())
    part.markt = abi.c_i8p()
    g.call("i3g_download", part, abi.SYNC_MARKERS)
    assert np.array_equal(got, whole["marky"])
    g.close()


@pytest.mark.parametrize("exact", [0, 1])
def test_marker_rheology_reads_what_it_needs(exact):
    """Power-law rocks (with and without activation energy) use the strain rate, a yielding rock the
    stress too, a Newtonian rock neither; positive strains of markers that do not yield turn negative."""
    bufs = []
    for side in range(2):
        p, mode, fx, buf = marker_setup("sphere13")
        rock = dict(zip(ROCK_FIELDS, buf.rocks))
        rock["n0"][:], rock["n1"][:] = 1e5, 1e35
        rng = np.random.default_rng(3)
        n = buf.f32["markx"].size
        buf.markt[:] = rng.integers(2, 4, n)
        for f, v in dict(nu=1e9, ss=1e4, mm=3.0).items():   # type 2: power law
            rock[f][2] = v
        for f, v in dict(nu=1e-3, dh=2e5, ss=1e4, mm=3.0, a0=1e6, a1=1e6).items():   # type 3: with activation energy, yielding
            rock[f][3] = v
        buf.f32["marke"][:] = rng.uniform(-1, 1, n)
        buf.f32["markv"][:] = 1e20
        par, fp = abi.make_params(mode, marker_exact=exact), abi.make_file_params(mode.files[0])
        fp.nubeg, fp.nuend = 1e5, 1e35
        dt = float(fx["fld_dt"][0])
        c = lib.Context(buf, par, fp) if side == 0 else O.Oracle(buf, par, fp)
        if side == 0:
            c.move_markers(dt)
        else:
            c.call("orc_move_markers", dt)
        c.download(abi.SYNC_ALL)
        c.close()
        bufs.append(buf)
    a, b = bufs
    for f in ("markx", "marky", "markz"):
        assert np.array_equal(a.f32[f], b.f32[f]), f
    assert np.array_equal(a.markt, b.markt)
    assert 0 < int((b.f32["marke"] > 0).sum()) < a.markt.size
    # strains grow by dt * strain rate, stored as FP32; viscosities pass through pow and exp
    np.testing.assert_allclose(a.f32["marke"], b.f32["marke"], rtol=2e-7, atol=0)
    np.testing.assert_allclose(a.f32["markv"], b.f32["markv"], rtol=2e-7)


@pytest.mark.parametrize("exact", [0, 1])
@pytest.mark.parametrize("which", ["all yield", "one yields", "power law alone", "none"])
def test_marker_rheology_for_every_kind_of_rock_table(which, exact):
    """Tables whose rocks all yield, one of them, none but with power-law creep, and none that reads an
    invariant: each has its own kernel.  Positions as the oracle's to the bit, strains within their FP32
    rounding, viscosities through pow and exp."""
    bufs = []
    for side in range(2):
        p, mode, fx, buf = marker_setup("sphere13")
        rock = dict(zip(ROCK_FIELDS, buf.rocks))
        rock["n0"][:], rock["n1"][:] = 1e5, 1e35
        rng = np.random.default_rng(6)
        n = buf.f32["markx"].size
        buf.markt[:] = rng.integers(2, 4, n)
        for t in (2, 3):
            for f, v in dict(nu=1e21, dh=0.0, dv=0.0, ss=0.0, mm=1.0, a0=0.0, a1=0.0, b0=0.0, b1=0.0).items():
                rock[f][t] = v
            if which == "all yield" or (which == "one yields" and t == 3):
                rock["a0"][t] = rock["a1"][t] = 1e6
                rock["b0"][t] = rock["b1"][t] = 0.1
            if which == "power law alone" and t == 3:
                rock["nu"][t], rock["ss"][t], rock["mm"][t] = 1e9, 1e4, 3.0
        buf.f32["marke"][:] = rng.uniform(-1, 1, n)
        buf.f32["markv"][:] = 1e20
        par, fp = abi.make_params(mode, marker_exact=exact), abi.make_file_params(mode.files[0])
        fp.nubeg, fp.nuend = 1e5, 1e35
        dt = float(fx["fld_dt"][0])
        c = lib.Context(buf, par, fp) if side == 0 else O.Oracle(buf, par, fp)
        if side == 0:
            c.move_markers(dt)
        else:
            c.call("orc_move_markers", dt)
        c.download(abi.SYNC_ALL)
        c.close()
        bufs.append(buf)
    a, b = bufs
    for f in ("markx", "marky", "markz"):
        assert np.array_equal(a.f32[f], b.f32[f]), f
    if "yield" in which:
        assert int((b.f32["marke"] > 0).sum()) > 0
    np.testing.assert_allclose(a.f32["marke"], b.f32["marke"], rtol=2e-7, atol=0)
    np.testing.assert_allclose(a.f32["markv"], b.f32["markv"], rtol=2e-7)


@pytest.mark.parametrize("factor", [None, 0.5])
@pytest.mark.parametrize("scale", [1e-2, 1.0, 30.0])
def test_heat_from_uncoupled_to_stiff(scale, factor):
    """Steps far below and far above the cells' diffusion time (level 0 alone, and all levels), with
    the boundary rows' own factors and with 1/2.  The matrix has row sums rho cp / dt, so two solutions
    with relative residuals 1e-13 agree to a few 1e-12; both are stored as FP32."""
    out = []
    for side in range(2):
        p, mode, fx, _ = marker_setup("sphere13")
        if factor is not None:
            b = p.bond
            heat = (b["row"] >= 8 * p.nodenum) & (b["partner1"] > 0)
            assert heat.sum() > 100
            b["k"][heat] = factor
        buf = abi.ModelBuffers(p)
        par, fp = abi.make_params(mode, heat_rtol=1e-13), abi.make_file_params(mode.files[0])
        fp.maxtkstep = 1e9
        dt = float(fx["fld_dt"][0]) * scale
        c = lib.Context(buf, par, fp) if side == 0 else O.Oracle(buf, par, fp)
        if side == 0:
            c.heat(0, dt)
            assert c.stats()["heat_rel"] <= 1e-13
        else:
            c.call("orc_heat", (O.C.c_double * 1)(dt))
        c.download(abi.SYNC_ALL)
        c.close()
        out.append(buf.f32["tk"].copy())
    assert np.all(np.isfinite(out[1]))
    np.testing.assert_allclose(out[0], out[1], rtol=2e-7, atol=0)


def _heat(edit, dt_scale, side, **kw):
    """One heat step of the 13^3 case, dt_scale times its time step, on the GPU (side 0) or the oracle."""
    p, mode, fx, _ = marker_setup("sphere13")
    edit(p)
    buf = abi.ModelBuffers(p)
    par, fp = abi.make_params(mode, heat_rtol=kw.pop("heat_rtol")), abi.make_file_params(mode.files[0])
    for f, v in kw.items():
        setattr(par, f, v)
    fp.maxtkstep = 1e30
    dt = float(fx["fld_dt"][0]) * dt_scale
    c = lib.Context(buf, par, fp) if side == 0 else O.Oracle(buf, par, fp)
    stats = None
    if side == 0:
        c.heat(0, dt)
        stats = c.stats()
    else:
        c.call("orc_heat", (O.C.c_double * 1)(dt))
    c.download(abi.SYNC_ALL)
    c.close()
    return buf.f32["tk"].copy(), stats


def test_heat_with_a_node_without_heat_capacity():
    """A node with rho cp = 0 makes the largest k / (rho cp) infinite: the stiff step takes as many cycles as
    with a heat capacity that is merely tiny there."""
    cycles = []
    for cp in (1e-9, 0.0):
        def edit(p):
            nx, ny, nz = p.shape
            p.nodes["ht"][:] = 0
            p.nodes["cp"][(nz // 2 * nx + nx // 2) * ny + ny // 2] = cp
        got, stats = _heat(edit, 1e3, 0, heat_rtol=1e-10, frictyn=0)
        assert np.all(np.isfinite(got)) and stats["heat_rel"] <= 1e-10
        cycles.append(stats["heat_cycles"])
    assert abs(cycles[1] - cycles[0]) <= 1, cycles


@pytest.mark.parametrize("n,multinum,stretch", [(65, 4, 0.3), (57, 4, 0.4), (41, 3, 0.3)])
def test_heat_on_stretched_grids(n, multinum, stretch):
    """Steps of 3 and 10 diffusion times of the mean cell, with cells at the walls that stay narrow on every
    level: solved in at most half as many cycles again as a V-cycle with 16 sweeps on the coarsest level
    takes (9 to 18)."""
    p, spec = model.sinking_sphere(n=n, mnum=1, multinum=multinum, stretch=stretch)
    mode = config.Mode(multinum=multinum, multinnn=((2,) * multinum + (0,), (2,) * multinum + (4,)), nubeg=1e18, nuend=1e24,
                       files=[config.OutFile("o.prn", maxxystep=1e3, nubeg=1e18, nuend=1e24, multinum=multinum, multinum2=multinum)])
    g = lib.Context(abi.ModelBuffers(p), abi.make_params(mode, heat_rtol=1e-10), abi.make_file_params(mode.files[0]))
    g.call("i3g_prepare")
    h = 1e5 / (n - 1)
    for times in (3, 10):
        g.heat(0, times * h * h / 1e-6)
        st = g.stats()
        assert st["heat_rel"] <= 1e-10 and st["heat_cycles"] <= 27, (times, st["heat_cycles"])
    g.close()


@pytest.mark.parametrize("t0koef", [1.0, 0.8, 1.3])
@pytest.mark.parametrize("scale", [0.1, 3.0])
def test_heat_of_strong_contrasts(scale, t0koef):
    """Good conductors (k and rho cp 1000 times larger) beside poor ones node by node: rows couple more strongly
    than their own k / (rho cp) says, with and without damping.  The matrix has row sums rho cp / dt of
    ratio 1000, so two solutions with relative residuals 1e-13 agree to a few 1e-9; both are stored as FP32."""
    def edit(p):
        nx, ny, nz = p.shape
        z, x, y = np.meshgrid(np.arange(nz), np.arange(nx), np.arange(ny), indexing="ij")
        good = ((x + y + z) & 1).reshape(-1) == 1
        for f in ("kt", "cp"):
            p.nodes[f] = np.where(good, 1000 * p.nodes[f], p.nodes[f]).astype(np.float32)
    got, stats = _heat(edit, scale, 0, heat_rtol=1e-13, t0koef=t0koef)
    assert stats["heat_rel"] <= 1e-13
    want, _ = _heat(edit, scale, 1, heat_rtol=1e-13)
    assert np.all(np.isfinite(want))
    np.testing.assert_allclose(got, want, rtol=2e-7, atol=0)


@pytest.mark.parametrize("cin,cout", [(32, 32), (32, 64), (64, 32), (64, 64), (64, 128), (128, 64), (128, 128)])
@pytest.mark.parametrize("dims", [(1, 1, 1), (10, 11, 14), (15, 17, 19), (27, 25, 29)])
def test_wide_convolutions_for_every_channel_split(dims, cin, cout):
    """1, 20, 53 and 190 tiles of 128 rows: 16 or 32 output channels per block, or the whole width.
    FP32 sums of 27 * cin <= 3456 products against FP64: relative error far below 27 cin 2^-24 = 2e-4;
    2e-5 of the largest output, as a random-sign sum of that length keeps."""
    rng = np.random.default_rng(cin * 1000 + cout)
    x = U.bf16(rng.normal(size=dims + (cin,)))
    w = U.bf16(rng.normal(0, 1 / np.sqrt(27 * cin), size=(27, cout, cin)))
    b = rng.normal(0, 0.1, size=cout).astype(np.float32)
    rows = np.pad(x, ((1, 1), (1, 1), (1, 1), (0, 0))).reshape(-1, cin)
    out = warmstart.conv_host(cin, cout, dims, U.bf16_bits(rows), U.bf16_bits(w), b, None, relu=False)
    got = out.reshape(dims[0] + 2, dims[1] + 2, dims[2] + 2, cout)
    inner = got[1:-1, 1:-1, 1:-1].copy()
    ref = U.conv3(x, w, b.astype(np.float64))
    assert np.max(np.abs(inner - ref)) <= 2e-5 * np.max(np.abs(ref)) + 1e-6
    got[1:-1, 1:-1, 1:-1] = 0
    assert not np.any(got)   # halo rows are not written


@pytest.mark.parametrize("name", ["sphere17", "stretch17"])
def test_fp32_cycles_of_every_tail_and_transfer(name, monkeypatch):
    """The FP32 cycle with the coarsest levels on chip and compact transfers, with the general tail,
    and with one launch per pass and the general transfers differs by rounding only: the solves need
    the same number of cycles within one in ten and agree to the solver's tolerance."""
    sols, cycles = [], []
    for env in ({}, {"I3G_SMTAIL": "0"}, {"I3G_FUSE": "0"}):
        for k in ("I3G_SMTAIL", "I3G_FUSE"):
            monkeypatch.delenv(k, raising=False)
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        p, mode, _ = golden(name)
        par = abi.make_params(mode, stokes_rtol=1e-10, stokes_maxcyc=3000, precision=1, krylov=8)
        g = lib.Context(abi.ModelBuffers(p), par, abi.make_file_params(mode.files[0]))
        g.stokes(0, 1e30)
        cycles.append(g.stats()["stokes_cycles"])
        sols.append(g.get(abi.A_SOL, 0, 4 * cases.level_sizes(p, mode.multinum)[0]).reshape(-1, 4))
        g.close()
    for q in (1, 2):
        assert abs(cycles[q] - cycles[0]) <= 1 + cycles[0] // 10, cycles
        for k in (1, 2, 3):
            assert np.linalg.norm(sols[q][:, k] - sols[0][:, k]) <= 1e-6 * np.linalg.norm(sols[0][:, k])


@pytest.mark.parametrize("shape,multinum,widths", [((23, 23, 23), 1, [4]), ((21, 21, 21), 2, [4, 4]), ((23, 23, 23), 2, [4, 4]), ((43, 21, 23), 3, [4, 4, 5]),
                                                   ((27, 43, 35), 3, [4, 4, 5]), ((51, 51, 51), 3, [4, 4, 5])])
def test_fp32_transfers_are_compact_on_every_grid(shape, multinum, widths, capfd, monkeypatch):
    """Coarse lines that gather from four or five fine ones, on grids whose FP32-rounded lines leave weights of
    1e-6 at coinciding points: every level takes the compact transfers, and the FP32 cycle preconditions as
    with the general ones (one launch per pass): cycles within one in ten, solutions to the tolerance."""
    sols, cycles = [], []
    for fuse in ("1", "0"):
        monkeypatch.setenv("I3G_FUSE", fuse)
        monkeypatch.setenv("I3G_TRACE", "1")
        p, mode = _random_box(shape, multinum, seed=11)
        z, x, y = np.meshgrid(*(np.linspace(0, 1, n) for n in (shape[2], shape[0], shape[1])), indexing="ij")
        eta = (1e21 * np.exp(1.5 * np.sin(5 * x + 2 * y) * np.cos(4 * z - y))).astype(np.float32).reshape(-1)
        for f in ("nu", "nxx", "nxy", "nxz", "nyz"):
            p.nodes[f] = eta.copy()
        par = abi.make_params(mode, stokes_rtol=1e-10, stokes_maxcyc=3000, precision=1, krylov=8)
        capfd.readouterr()
        g = lib.Context(abi.ModelBuffers(p), par, abi.make_file_params(mode.files[0]))
        seen = [int(s.split(": ")[2].split()[0]) for s in capfd.readouterr().err.splitlines() if "FP32 transfers" in s]
        assert seen == (widths if fuse == "1" else [0] * multinum)
        monkeypatch.delenv("I3G_TRACE")
        g.stokes(0, 1e30)
        cycles.append(g.stats()["stokes_cycles"])
        sols.append(g.get(abi.A_SOL, 0, 4 * p.nodenum).reshape(-1, 4))
        g.close()
    assert abs(cycles[1] - cycles[0]) <= 1 + cycles[0] // 10, cycles
    for k in (1, 2, 3):
        assert np.linalg.norm(sols[1][:, k] - sols[0][:, k]) <= 1e-6 * np.linalg.norm(sols[0][:, k])


@pytest.mark.parametrize("krylov", [8, 0])
def test_viscosity_limits_of_the_next_output_row(krylov):
    """Another row of the output plan may set other viscosity limits, whose mean scales the FP32 cycle: a solve
    after the change takes as many cycles as in a context that had these limits from the start."""
    p, mode, _ = golden("sphere17")
    par = abi.make_params(mode, stokes_rtol=1e-8, stokes_maxcyc=3000, precision=1, krylov=krylov, warm_start=0)
    wide, narrow = abi.make_file_params(mode.files[0]), abi.make_file_params(mode.files[0])
    wide.nubeg, wide.nuend = 1e12, 1e24
    narrow.nubeg, narrow.nuend = 1e20, 1e24
    cycles = []
    for first in (narrow, wide):
        g = lib.Context(abi.ModelBuffers(p), par, first)
        g.stokes(0, 1e30)
        g.set_file_params(narrow)
        g.stokes(0, 1e30)
        cycles.append(g.stats()["stokes_cycles"])
        g.close()
    assert abs(cycles[1] - cycles[0]) <= 1, cycles
