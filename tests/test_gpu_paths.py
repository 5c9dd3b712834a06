"""The paths a size, a row length or a step count selects, against the general
ones: device rows padded to 16 bytes, short z chunks, accumulators added several
steps at a time, the one-pass Mur faces, the heat step's paired doses and its
integer dose add, bubbles in one-warp blocks.  Wherever both paths perform the
same operations on every value the comparison is bit for bit."""
import ctypes as C

import numpy as np
import pytest

from bubbledynamics_gb300 import abi, api, presets

pytestmark = pytest.mark.gpu

FIELDS = ("p_final", "peak", "energy", "Q", "dft_re", "dft_im")


def same(a, b, msg):
    for k in FIELDS:
        if k in a:
            np.testing.assert_array_equal(a[k], b[k], err_msg="%s: %s" % (msg, k))


def burst(nx, ny, nz, steps):
    return presets.cfg1(nx, ny, nz, steps, precision=abi.BD_F32)


def layers(nx, nz, periods=1, precision=abi.BD_F32):
    p = presets.ref_W_mini(precision, Nxy=nx, Nz=nz, loop1_periods=1, periods=periods)
    return p


def mapped(nx, ny, nz, steps):
    """Water and liver mixed cell by cell (0 and 1 relaxation process)."""
    p = presets.cfg1(nx, ny, nz, steps, precision=abi.BD_F32, heterogeneity=False)
    p.medium.n_materials = 2
    p.medium.mat[1] = presets.slab_materials(1.0e6)[2]
    p.medium.mat[0].n_relax = 0
    p.set_material_map((np.random.default_rng(3).random((nz, ny, nx)) < 0.5).astype(np.uint8))
    return p


@pytest.mark.parametrize("nx", [33, 34, 35, 61, 65, 67])
def test_padded_rows_equal_the_plain_kernel(ctx, nx):
    """Row lengths on either side of the 32- and 64-cell tiles and of every remainder
    modulo four: the padded two-cell variants and the default give the plain
    kernel's bits (c map, material map, mirror and Mur faces with the DFT)."""
    for make in (lambda: burst(nx, 27, 41, 45), lambda: mapped(nx, 27, 41, 45), lambda: layers(nx, 40)):
        base = None
        for v in (0, -1, 24, 25, 26, 27, 28):
            p = make()
            p.params.tile_variant = v
            r = ctx.westervelt(p)
            if v >= 0:
                assert r["tile_variant"] == v
            if base is None:
                base = r
                assert np.abs(r["p_final"]).max() > 0
            else:
                same(r, base, "nx %d, variant %d" % (nx, v))


@pytest.mark.parametrize("nx", [44, 45, 46])
def test_fp64_rows_with_a_c_map(ctx, nx):
    """FP64 rows of 16-byte vectors whose float c map's rows are none (nx = 46): the default
    is the plain kernel there, a TMA variant is refused, and the bits are the same."""
    def make(v):
        p = presets.cfg1(nx, 27, 41, 40, precision=abi.BD_F64)
        p.params.tile_variant = v
        return p
    base = ctx.westervelt(make(0))
    assert np.abs(base["p_final"]).max() > 0
    same(ctx.westervelt(make(-1)), base, "default")
    if nx % 4 == 0:
        same(ctx.westervelt(make(17)), base, "variant 17")
    else:
        with pytest.raises(api.BDError) as e:
            ctx.westervelt(make(17))
        assert e.value.status == abi.BD_ERR_INVALID_ARG


@pytest.mark.parametrize("nz", [8, 9, 15, 17, 50])
def test_short_chunks_equal_the_plain_kernel(ctx, nz):
    """Grids that do not fill one wave run in chunks of two planes or more."""
    base = None
    for v in (0, 17, 19, 21, 23, -1):
        p = burst(40, 36, nz, 40)
        p.params.tile_variant = v
        r = ctx.westervelt(p)
        base = base or r
        same(r, base, "nz %d, variant %d" % (nz, v))


@pytest.mark.parametrize("mode", [abi.BD_ENERGY_P2, abi.BD_ENERGY_DPDT2])
def test_deferred_accumulators_in_any_pieces(ctx, mode):
    """Windows that open and close between the steps that accumulate, advanced in
    pieces of every length: the bits of the one-cell kernel, which accumulates
    every step (variant 17), and of the run in one piece with graphs."""
    def make(v):
        p = layers(28, 40)
        p.params.energy_mode = mode
        n = p.params.n_steps
        p.params.peak_start, p.params.peak_end = 3, n - 7
        p.params.energy_start, p.params.energy_end = 22, 137
        p.params.dft_start, p.params.dft_len = 101, 61
        p.params.tile_variant = v
        return p
    base = ctx.westervelt(make(17))
    assert np.abs(base["dft_re"]).max() > 0 and base["energy"].max() > 0
    for v in (19, 21, 23):
        same(ctx.westervelt(make(v)), base, "one run, variant %d" % v)
        p = make(v)
        with ctx.westervelt_session(p) as s:
            k, left = 1, p.params.n_steps
            while left:
                n = min(k % 13 + 1, left)
                s.advance(n)
                left -= n
                k += 1
            same(s.finish(), base, "pieces, variant %d" % v)


@pytest.mark.parametrize("precision", [abi.BD_F32, abi.BD_F64])
@pytest.mark.parametrize("n_layers", [1, 2, 5, 8])
def test_mur_layer_counts(ctx, oracle, precision, n_layers):
    """The one-pass Mur faces with other layer counts than the reference's three
    (the x+, y+ and z+ runs meet in the corners): 1e-9 of the FP64 oracle, the
    1e-5 field tolerance in FP32."""
    p = layers(26, 44, precision=precision)
    p.grid.mur_layers = n_layers
    q = layers(26, 44, precision=abi.BD_F64)
    q.grid.mur_layers = n_layers
    got, exp = ctx.westervelt(p), oracle.westervelt(q)
    for k in ("p_final", "peak", "Q"):
        a, b = np.asarray(got[k], np.float64), exp[k].reshape(got[k].shape)
        assert np.linalg.norm(a - b) <= (1e-9 if precision == abi.BD_F64 else 1e-5) * np.linalg.norm(b), k


@pytest.mark.parametrize("precision", [abi.BD_F32, abi.BD_F64])
@pytest.mark.parametrize("nz,n_layers,plane", [(12, 3, 8), (12, 4, 8), (16, 8, 8), (12, 4, 10), (13, 8, 12)])
def test_mur_z_runs_that_meet(ctx, oracle, precision, nz, n_layers, plane):
    """Mur on both z faces, z- up to a source plane on either side of the first z+ layer: one
    plane between the runs, none, and cells in both.  The oracle's order, 1e-9 of it in
    FP64 and the 1e-5 field tolerance in FP32, in repeated runs the same bits."""
    def make(precision):
        p = layers(26, 40, precision=precision)
        p.grid.nz, p.grid.mur_layers, p.source.plane_iz = nz, n_layers, plane
        p.params.q_mode, p.params.n_dft = abi.BD_Q_NONE, 0
        p.params.n_steps, p.params.peak_start, p.params.peak_end = 60, 5, 50
        p.params.energy_start, p.params.energy_end = 10, 55
        return p
    want = ("p_final", "peak", "energy")
    got = ctx.westervelt(make(precision), want=want)
    for _ in range(3):
        same(ctx.westervelt(make(precision), want=want), got, "again")
    exp = oracle.westervelt(make(abi.BD_F64))
    for k in want:
        a, b = np.asarray(got[k], np.float64), np.asarray(exp[k]).reshape(got[k].shape)
        assert plane > nz - n_layers or np.abs(b).max() > 0      # a z+ layer over the source plane leaves no wave
        assert np.linalg.norm(a - b) <= (1e-9 if precision == abi.BD_F64 else 1e-5) * np.linalg.norm(b), k


@pytest.mark.parametrize("face", [1, 3, 4, 5])
def test_mur_layers_that_fill_an_axis_are_refused(ctx, face):
    """Eight layers on an axis of eight cells have no inner neighbour: the run would read cells
    in front of (z-: behind) the field.  Nine cells are enough."""
    def make(cells):
        nx, ny, nz = (cells if face == 1 else 12), (cells if face == 3 else 12), (cells if face > 3 else 24)
        p = presets.cfg1(nx, ny, nz, 4, heterogeneity=False)
        p.grid.face[face] = abi.BD_FACE_MUR
        p.grid.mur_layers = 8
        p.source.kind = abi.BD_SRC_NONE
        return p
    with pytest.raises(api.BDError) as e:
        ctx.westervelt(make(8))
    assert e.value.status == abi.BD_ERR_INVALID_ARG and "Mur layers" in str(e.value)
    assert not ctx.westervelt(make(9), want=("p_final",))["p_final"].any()


@pytest.mark.parametrize("nx", [40, 41])
def test_two_processes_with_a_c_map(ctx, nx):
    """Two relaxation processes in the semi-implicit scheme on a c map, strong enough that a
    rounding of their coefficients shows: every variant gives the plain kernel's bits."""
    base = None
    for v in (0, 17, 18, 19, 21, 23, 24, 26, 28):
        if nx % 4 and 8 <= v < 24:
            continue
        p = burst(nx, 34, 45, 60)
        mt = p.medium.mat[0]
        mt.n_relax = 2
        for k, (c, tau) in enumerate(((60.0, 1.0e-7), (45.0, 3.0e-8))):
            mt.relax_c[k], mt.relax_tau[k] = c, tau
        p.params.tile_variant = v
        r = ctx.westervelt(p)
        base = base or r
        assert 0 < np.abs(base["p_final"]).max() < 1e8
        same(r, base, "nx %d, variant %d" % (nx, v))


@pytest.mark.parametrize("nx", [33, 35])
def test_checkpoint_between_padded_and_plain_rows(ctx, nx):
    """A checkpoint has rows of nx cells whatever the device's: one taken on padded
    rows continues on the plain kernel's, and the other way round."""
    whole = ctx.westervelt(layers(nx, 40))
    for first, second in ((-1, 0), (0, -1)):
        a, b = layers(nx, 40), layers(nx, 40)
        a.params.tile_variant, b.params.tile_variant = (first, second)
        if first == -1:
            a.params.tile_variant = 28
        if second == -1:
            b.params.tile_variant = 28
        with ctx.westervelt_session(a) as s:
            s.advance(63)
            blob = s.checkpoint()
        with ctx.westervelt_session(b) as s:
            s.restore(blob)
            s.advance(a.params.n_steps - 63)
            same(s.finish(), whole, "%d -> %d" % (first, second))


@pytest.mark.parametrize("precision", [abi.BD_F32, abi.BD_F64])
def test_constants_of_successive_solves(precision):
    """Solves of two media in turn on one context, whose constants take the block that the
    solve before left: each gives the bits of a fresh context, so every upload is in
    place before the kernel that derives the coefficients reads it."""
    def make(k):
        p = layers(24, 40, precision=precision)
        for m in range(p.medium.n_materials):
            p.medium.mat[m].c0 *= 1.0 + 0.01 * k
        p.params.n_steps = 20
        return p
    fresh = []
    for k in (0, 1):
        with api.Context(0) as c:
            fresh.append(c.westervelt(make(k), want=("p_final",)))
    assert np.abs(fresh[0]["p_final"] - fresh[1]["p_final"]).max() > 0
    with api.Context(0) as c:
        for i in range(24):
            same(c.westervelt(make(i % 2), want=("p_final",)), fresh[i % 2], "solve %d" % i)


# --------------------------------------------------------------------------- heat
def thermal(nx, ny, nz, steps, precision=abi.BD_F32, material_map=False):
    k = presets.ref_T_mini_constants(Nxy=nx, Nz=nz, legs=2)
    p = presets.make_ref_T(k, precision=precision)
    p.thermal.ny = ny
    if material_map:
        p.set_material_map((np.random.default_rng(5).random((nz, ny, nx)) < 0.5).astype(np.uint8))
    p.set_spots([0, 3, -2], [0, 1, -4], [steps // 3, steps // 3, steps - 2 * (steps // 3)])
    Q = presets.gaussian_focus_Q((nz, ny, nx), (nz // 2, ny // 2, nx // 2), (3.0, 2.0, 2.0), 4.0e7)
    return p, Q


@pytest.mark.parametrize("precision", [abi.BD_F32, abi.BD_F64])
@pytest.mark.parametrize("nx,ny,nz,steps", [(3, 3, 3, 5), (9, 11, 7, 1), (13, 9, 70, 2), (66, 17, 8, 67), (131, 8, 9, 64)])
def test_heat_run_equals_single_steps(ctx, precision, nx, ny, nz, steps):
    """Doses added for two steps at once, padded rows and every chunk length, against
    the same run advanced one step at a time (each step its own dose)."""
    for material_map in (False, True):
        p, Q = thermal(nx, ny, nz, steps, precision, material_map)
        one = ctx.heat(p.thermal, Q, p.traj)
        s = ctx.heat_slab(p.thermal, Q, p.traj, 0, nz)
        for _ in range(steps):
            s.advance(1)
        got = s.finish()
        s.close()
        np.testing.assert_array_equal(one["T"], got["T"])
        np.testing.assert_array_equal(one["dose"], got["dose"])


@pytest.mark.parametrize("nx,ny,nz", [(66, 600, 40), (67, 599, 41), (253, 160, 83)])
def test_heat_dose_free_kernel(ctx, nx, ny, nz):
    """Grids large enough for chunks of four planes and more, whose steps without the dose
    take their own kernel: the bits of single steps, which the general kernel runs."""
    p, Q = thermal(nx, ny, nz, 5)
    one = ctx.heat(p.thermal, Q, p.traj)
    s = ctx.heat_slab(p.thermal, Q, p.traj, 0, nz)
    for _ in range(5):
        s.advance(1)
    got = s.finish()
    s.close()
    np.testing.assert_array_equal(one["T"], got["T"])
    np.testing.assert_array_equal(one["dose"], got["dose"])
    assert one["T"].max() > p.thermal.T_ref


def device_bytes(torch):
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_heat_run_memory():
    """An FP32 heating run holds 20 bytes a cell (two temperatures and the source in float, the
    dose in double) and a staging buffer of bounded size."""
    torch = pytest.importorskip("torch")
    with api.Context(0) as c:
        p, Q = thermal(34, 30, 12, 2)
        c.heat(p.thermal, Q, p.traj)                  # kernels loaded
        nx, ny, nz = 253, 250, 300
        p, Q = thermal(nx, ny, nz, 2)
        before = device_bytes(torch)
        s = c.heat_slab(p.thermal, Q, p.traj, 0, nz)
        held = before - device_bytes(torch)
        s.close()
    assert held <= 20 * 256 * ny * nz + (48 << 20)


def test_fields_through_several_staging_groups(ctx):
    """Source, start fields and results of a grid of several staging buffers: two steps
    match FP64 (the FP32 tolerance, 1e-5) and two slabs give the same bits; with no steps the
    start comes back, its temperatures in float around T_ref."""
    nx, ny, nz, steps = 255, 254, 150, 2
    p, Q = thermal(nx, ny, nz, steps)
    rng = np.random.default_rng(8)
    T0, D0 = 300.0 + 40.0 * rng.random((nz, ny, nx)), rng.random((nz, ny, nx))
    p.set_start(T0, D0)
    got = ctx.heat(p.thermal, Q, p.traj, n_slabs=1)
    two = ctx.heat(p.thermal, Q, p.traj, n_slabs=2)
    np.testing.assert_array_equal(got["T"], two["T"])
    np.testing.assert_array_equal(got["dose"], two["dose"])
    q, _ = thermal(nx, ny, nz, steps, abi.BD_F64)
    q.set_start(T0, D0)
    exp = ctx.heat(q.thermal, Q, q.traj)
    assert np.abs(got["T"] - exp["T"]).max() <= 1e-5 * 40.0
    np.testing.assert_allclose(got["dose"], exp["dose"], rtol=1e-5)
    q = presets.ThermalProblem("start", p.thermal, p.traj, p._keep)
    q.set_spots([0], [0], [0])
    back = ctx.heat(q.thermal, Q, q.traj)
    np.testing.assert_array_equal(back["dose"], D0)
    np.testing.assert_array_equal(back["T"], p.thermal.T_ref + (T0 - p.thermal.T_ref).astype(np.float32).astype(np.float64))


def test_heat_run_of_many_planes(ctx):
    """More planes than the four-cell kernel's six-plane chunks could number in a grid's z extent."""
    nx, ny, nz, steps = 6, 5, 400001, 3
    p, Q = thermal(nx, ny, nz, steps)
    q, _ = thermal(nx, ny, nz, steps, abi.BD_F64)
    got, exp = ctx.heat(p.thermal, Q, p.traj)["T"], ctx.heat(q.thermal, Q, q.traj)["T"]
    rise = np.abs(exp - q.initial_fields()[0]).max()
    assert rise > 1e-3
    assert np.abs(got - exp).max() <= 1e-5 * rise + 1e-9


@pytest.mark.parametrize("nx", [13, 14, 15])
def test_material_map_on_padded_rows(nx):
    """The cells between padded rows hold a material of the table whatever the block of the
    map last held: its bytes are 255 here (an FP64 run of no steps whose fields are all
    ones), an index far outside.  The bits of the run on a fresh context."""
    ny, nz = 10, 9                                           # 16 x 10 x 9 bytes
    p, Q = thermal(nx, ny, nz, 5, material_map=True)
    with api.Context(0) as c:
        fresh = c.heat(p.thermal, Q, p.traj)
    ones, _ = thermal(5, 6, 6, 3, abi.BD_F64)                # 180 doubles
    ones.set_spots([0], [0], [0])
    fill = np.full(180, 2 ** 64 - 1, np.uint64).view(np.float64).reshape(6, 6, 5)
    ones.set_start(fill, fill)
    with api.Context(0) as c:
        c.heat(ones.thermal, fill, ones.traj)
        got = c.heat(p.thermal, Q, p.traj)
    np.testing.assert_array_equal(got["T"], fresh["T"])
    np.testing.assert_array_equal(got["dose"], fresh["dose"])


def test_dose_add_is_the_fp64_sum(ctx):
    """One step onto doses of every magnitude, sign and kind: the bits of start + increment in
    double (the increment itself is the dose of the same step from zero)."""
    nx, ny, nz = 34, 30, 12
    p, Q = thermal(nx, ny, nz, 1)
    p.thermal.dose_init = 0
    inc = ctx.heat(p.thermal, Q, p.traj)["dose"]
    T0, _ = p.initial_fields()
    rng = np.random.default_rng(11)
    n = nx * ny * nz
    start = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-60, 60, n)) * np.where(rng.random(n) < 0.1, -1.0, 1.0)
    start *= np.median(inc[1:-1, 1:-1, 1:-1])
    start[:: 7] = (np.ldexp(1.0, rng.integers(0, 40, n)) * inc.reshape(-1) * (1.0 - 2.0 ** -53))[:: 7]   # next to a carry
    start[::101], start[1::101], start[2::101] = 0.0, np.inf, np.nan
    start[3::101], start[4::101], start[5::101] = 5e-324, 1e308, -0.0
    start = start.reshape(nz, ny, nx)
    p.set_start(T0, start)
    got = ctx.heat(p.thermal, Q, p.traj)["dose"]
    exp = start.copy()
    exp[1:-1, 1:-1, 1:-1] += inc[1:-1, 1:-1, 1:-1]
    np.testing.assert_array_equal(got, exp)


@pytest.mark.parametrize("steps", [1, 2])
@pytest.mark.parametrize("kelvin", [600.0, np.inf, np.nan])
def test_dose_add_of_a_rate_that_is_no_number(ctx, steps, kelvin):
    """Above 171 C the float rate is infinite: the dose becomes infinite (NaN for a NaN
    temperature) whatever it was, also between 2^128 and 2^157, where the exponents of an
    infinite increment and of the dose are as close as those the integer add takes."""
    nx, ny, nz = 18, 14, 11
    p, Q = thermal(nx, ny, nz, steps)
    start = np.ldexp(np.random.default_rng(2).uniform(1.0, 2.0, nx * ny * nz), np.arange(nx * ny * nz) % 60 + 110)
    start = start.reshape(nz, ny, nx)
    p.set_start(np.full((nz, ny, nx), kelvin), start)
    got = ctx.heat(p.thermal, Q, p.traj)["dose"]
    exp = start.copy()
    exp[1:-1, 1:-1, 1:-1] = np.nan if np.isnan(kelvin) else np.inf
    np.testing.assert_array_equal(got, exp)


@pytest.mark.parametrize("nx", [40, 41])
@pytest.mark.parametrize("steps", [1, 2, 65])
def test_noalloc_steps_equal_the_run(ctx, nx, steps):
    """The allocation-free run on vector and scalar rows: the allocating run's
    temperature bit for bit, its dose to the 2^-47 of a float pair."""
    torch = pytest.importorskip("torch")
    p, Q = thermal(nx, 23, 31, steps)
    th = p.thermal
    exp = ctx.heat(th, Q, p.traj)
    sx, sy, _ = api.trajectory_shifts(p.traj)
    shifts = np.ascontiguousarray(np.stack([sx, sy], axis=1).astype(np.int32))
    T0, D0 = p.initial_fields()
    hi = D0.astype(np.float32)
    pair = np.ascontiguousarray(np.stack([hi, (D0 - hi).astype(np.float32)], axis=-1))
    theta, q, dose = (torch.from_numpy(a).cuda() for a in ((T0 - th.T_ref).astype(np.float32), Q.astype(np.float32), pair))
    torch.cuda.synchronize()
    api.check(ctx.L.bd_heat_run_device_noalloc(ctx.h, C.byref(th), theta.data_ptr(), q.data_ptr(), dose.data_ptr(),
                                               shifts.ctypes.data, len(sx), None))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(th.T_ref + theta.cpu().numpy().astype(np.float64), exp["T"])
    d = dose.cpu().numpy().astype(np.float64).sum(-1)
    np.testing.assert_allclose(d, exp["dose"], rtol=2.0 ** -44)


# --------------------------------------------------------------------------- staging
def test_checkpoint_memory_of_padded_rows():
    """A checkpoint of padded rows goes through a staging buffer of bounded size, not one of all
    the DFT accumulators."""
    torch = pytest.importorskip("torch")
    p = layers(131, 200)
    w = p.params
    w.n_dft, w.dft_z_lo, w.dft_z_hi, w.dft_len, w.dft_start = 10, 0, 200, 20, 1
    w.tile_variant = 26
    with api.Context(0) as c, c.westervelt_session(p) as s:
        s.advance(20)
        before = device_bytes(torch)
        s.checkpoint()
        held = before - device_bytes(torch)
    assert held <= 48 << 20


def test_fields_through_several_staging_pieces(ctx):
    """Fields of padded rows larger than the staging buffer, in and out: the c map, the results
    and a checkpoint's blob are those of the plain kernel's rows."""
    out, blobs = [], []
    c = (1500.0 * (1.0 + 0.01 * np.random.default_rng(6).random((160, 250, 251)))).astype(np.float32)   # 40 MB a field
    p = presets.cfg1(251, 250, 160, 12, heterogeneity=False)
    p.set_c_map(c)
    for v in (0, 26):
        p.params.tile_variant = v
        with ctx.westervelt_session(p) as s:
            s.advance(12)
            blobs.append(s.checkpoint())
            out.append(s.finish(want=("p_final", "peak", "energy")))
    assert np.abs(out[0]["p_final"]).max() > 0
    same(out[1], out[0], "results")
    assert bytes(blobs[1]) == bytes(blobs[0])
    with ctx.westervelt_session(p) as s:
        s.restore(blobs[0])
        same(s.finish(want=("p_final", "peak", "energy")), out[0], "restored")


# --------------------------------------------------------------------------- bubbles
def test_bubbles_do_not_depend_on_the_batch(ctx):
    """One-warp blocks (batches that fit the resident lanes) and the one-thread-per-bubble
    schedule: a bubble's result is the same in a batch of any size."""
    med, ode = presets.cfg2_medium(), presets.cfg2_ode(t_end=2e-11)
    b = presets.cfg2_bubbles(257, seed=5)
    whole, _ = ctx.gilmore(med, b, ode)
    for n in (1, 31, 32, 33, 129):
        part, _ = ctx.gilmore(med, b[:n], ode)
        np.testing.assert_array_equal(part, whole[:n])
    ode.schedule = abi.BD_SCHEDULE_STATIC
    np.testing.assert_array_equal(ctx.gilmore(med, b, ode)[0], whole)


def test_bubbles_across_the_launch_shapes(ctx):
    """A batch larger than the resident lanes of any occupancy (2,048 threads a SM), on the
    persistent kernel and on four-warp blocks of the static one, against one-warp blocks."""
    torch = pytest.importorskip("torch")
    n = 2048 * torch.cuda.get_device_properties(0).multi_processor_count + 1
    med, ode = presets.cfg2_medium(), presets.cfg2_ode(t_end=1e-12)
    b = presets.cfg2_bubbles(n, seed=5)
    ends = np.concatenate([b[:150], b[-107:]])
    small, _ = ctx.gilmore(med, ends, ode)
    for schedule in (abi.BD_SCHEDULE_PERSISTENT, abi.BD_SCHEDULE_STATIC):
        ode.schedule = schedule
        r, _ = ctx.gilmore(med, b, ode)
        np.testing.assert_array_equal(np.concatenate([r[:150], r[-107:]]), small)


# --------------------------------------------------------------------------- DFT pass
@pytest.mark.parametrize("precision", [abi.BD_F32, abi.BD_F64])
@pytest.mark.parametrize("nx,n_dft", [(27, 1), (28, 4), (29, 5), (26, 16)])
def test_dft_pass(ctx, oracle, precision, nx, n_dft):
    """The DFT pass on odd and even planes (scalar and 16-byte accesses; the FP32 rows are
    padded), every remainder of its groups of four frequencies, a window that opens and
    closes inside a group of steps and planes that start off a 16-byte boundary: the
    bits of the run advanced one step at a time, and the FP64 oracle (1e-9 of the
    largest accumulator in FP64, the 1e-5 field tolerance in FP32)."""
    def make(precision):
        p = layers(nx, 40, precision=precision)
        w = p.params
        w.n_dft = n_dft
        for j in range(n_dft):
            w.dft_freq[j] = 1.0e6 * (j + 1)
        w.dft_start, w.dft_len = w.n_steps - 77, 73
        w.dft_z_lo, w.dft_z_hi = 3, 36
        return p
    whole = ctx.westervelt(make(precision), want=("p_final", "dft"))
    p = make(precision)
    with ctx.westervelt_session(p) as s:
        for _ in range(p.params.n_steps):
            s.advance(1)
        same(s.finish(want=("p_final", "dft")), whole, "step by step")
    same(ctx.westervelt_slabs(make(precision), 2, want=("p_final", "dft")), whole, "two slabs (rows of nx cells)")
    exp = oracle.westervelt(make(abi.BD_F64))
    tol = 1e-9 if precision == abi.BD_F64 else 1e-5
    for k in ("dft_re", "dft_im"):
        a, b = np.asarray(whole[k], np.float64), np.asarray(exp[k]).reshape(whole[k].shape)
        assert np.abs(b).max() > 0
        assert np.linalg.norm(a - b) <= tol * np.sqrt(np.linalg.norm(exp["dft_re"]) ** 2 + np.linalg.norm(exp["dft_im"]) ** 2), k


@pytest.mark.parametrize("n_relax", [0, 1, 2, 3])
def test_fp64_kernels_by_relaxation_count(ctx, n_relax):
    """The FP64 TMA kernels compiled for 0, 1 and 2 relaxation processes, and the one that
    reads the count, give the plain kernel's bits (plane materials, Mur, the DFT)."""
    base = None
    for v in (0, 8, 9, 16, 17, 18, -1):
        p = layers(28, 40, precision=abi.BD_F64)
        for m in range(p.medium.n_materials):
            mt = p.medium.mat[m]
            for k in range(mt.n_relax, n_relax):
                mt.relax_tau[k], mt.relax_c[k] = 1.0e-8 * (k + 1), 1.0
            mt.n_relax = n_relax if m % 2 == 0 else min(n_relax, 1)
        p.params.tile_variant = v
        r = ctx.westervelt(p)
        base = base or r
        same(r, base, "%d processes, variant %d" % (n_relax, v))
