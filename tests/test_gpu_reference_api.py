"""The reference-named entry points (fmm_construct ... fmm_ext) driven
through the reference's globals, as src/photoNs.c:97-116 drives them, and
the batched operators and the FP64 direct sum against the oracle."""
import contextlib
import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


def rel_err(a, b, p):
    """Per-particle relative error |a-b|/|b|.  Where the net force cancels
    below 1e-4 of one nearest-neighbour pair force m/D^2 (D = L/N^(1/3);
    exact lattices cancel to ~1e-5 of it), the error is taken relative to
    that floor instead of the cancelled value."""
    nb = np.linalg.norm(b, axis=1)
    spacing = p["boxsize"] / np.cbrt(b.shape[0])
    floor = 1e-4 * p["mass"] / spacing ** 2
    return np.linalg.norm(a - b, axis=1) / np.maximum(nb, floor)


@pytest.mark.parametrize("name", ["grid16_leaf16", "nfw16_leaf8"])
def test_driver_sequence_matches_reference(ph, name):
    g = load_golden(name)
    ref = ph.Reference()
    ref.setup(g["pos_in"], g["p"])
    acc_task = ref.force_pass()
    part = ref.part()
    # part[] permuted into tree order, like the reference
    assert np.array_equal(part["pos"], g["pos_tree"])
    assert rel_err(acc_task, g["acc_task"], g["p"]).max() <= 1e-10
    assert rel_err(part["acc"], g["acc"], g["p"]).max() <= 1e-10
    c = ref.counters()
    assert c["idxP2P"] == g["counters"][0]
    assert c["idxM2L"] == g["counters"][1]
    assert c["walk_m2l_count"] == g["counters"][2]
    assert c["p2p_count_remote"] == g["counters"][3]
    ref.deconstruct()


def _pm_golden():
    import glob
    import os
    from conftest import GOLDEN
    return sorted(glob.glob(os.path.join(GOLDEN, "pm", "*.npz")))


@pytest.mark.parametrize("path", _pm_golden(), ids=lambda p: p.rsplit("/", 1)[-1][:-4])
def test_partmesh_matches_reference_pm(ph, path):
    """partmesh_thread() on the reference's globals against the reference's
    own partmesh.c outputs (cuFFT against a direct DFT: last bits)."""
    z = np.load(path)
    L, N, rs, m = z["params"]
    ref = ph.Reference()
    ref.setup(z["pos"], dict(boxsize=L, theta=0.5, rs=rs, rcut=4.5 * rs, eps=0.0, mass=m, maxleaf=16))
    got = ref.pm(int(N))
    want = z["acc_pm"]
    assert np.abs(got - want).max() <= 1e-10 * np.abs(want).max()


def test_driver_sequence_with_pm_thread(ph):
    """The driver's step with the PM on its own thread beside fmm_task: the
    FMM result is unchanged and acc_pm is the PM of the tree-ordered part[]."""
    import pm_oracle
    g = load_golden("grid16_leaf16")
    ref = ph.Reference()
    ref.setup(g["pos_in"], g["p"])
    nside = 16
    ref.force_pass(pm_nside=nside)
    part = ref.part()
    assert rel_err(part["acc"], g["acc"], g["p"]).max() <= 1e-10
    p = g["p"]
    want = pm_oracle.pm_force(part["pos"], p["boxsize"], nside, p["rs"], p["mass"])
    assert np.abs(part["acc_pm"] - want).max() <= 1e-10 * np.abs(want).max()
    ref.deconstruct()


def test_operators_match_oracle(ph, port):
    rng = np.random.default_rng(2)
    n = 64
    d = rng.normal(size=(n, 3)) * 4
    M = rng.normal(size=(n, 20))
    L0 = rng.normal(size=(n, 20))
    rs = 1.7
    got = ph.op_batch("m2l", d, M, L0, rs)
    want = np.array([L0[i] + port.m2l(d[i], M[i], rs) for i in range(n)])
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
    got = ph.op_batch("m2m", d, M, L0)
    want = np.array([L0[i] + port.m2m(d[i], M[i]) for i in range(n)])
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
    got = ph.op_batch("l2l", d, M, L0)
    want = np.array([L0[i] + port.l2l(d[i], M[i]) for i in range(n)])
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


def test_direct_sum_matches_oracle(ph, port, ics):
    pos, p = ics.make("nfw128", nside=24)
    targets = np.random.default_rng(4).choice(pos.shape[0], 500, replace=False).astype(np.int32)
    got = ph.direct_sum(pos, p, targets)
    want = port.direct_sum(pos, p, targets, nthreads=8)
    assert rel_err(got, want, p).max() <= 1e-10


def test_fp32_fma_probe_runs(ph):
    v = ph.fp32_fma_peak(2048)
    assert 1.0 < v < 1000.0


IMAGE_SHIFTS = [(mi, mj, mk) for mi in (-1, 0, 1) for mj in (-1, 0, 1) for mk in (-1, 0, 1) if (mi, mj, mk) != (0, 0, 0)]


@pytest.mark.parametrize("name", ["grid16_leaf16", "nfw16_leaf8"])
def test_fmm_remote_per_image_then_host_downward(ph, name):
    """fmm_ext's own sequence spelled out through the exported entry points
    (src/fmm.c:1028-1070): after fmm_task, fmm_remote(0, shift) for the 26
    image shifts, then the host walk_l2l from the root and l2p of every
    leaf.  The accelerations and counters equal the reference's pass (the
    nfw16 fixture has local and image M2L, so the host downward pass carries
    the GPU's local expansions)."""
    import ctypes as C
    g = load_golden(name)
    p = g["p"]
    ref = ph.Reference()
    ref.setup(g["pos_in"], p)
    lib = ref.lib
    lib.walk_l2l.argtypes = [C.c_int]
    lib.l2p.argtypes = [C.c_int]
    lib.fmm_construct()
    lib.fmm_prepare()
    lib.fmm_task()
    part = ref.part()
    assert rel_err(part["acc"].copy(), g["acc_task"], p).max() <= 1e-10
    for s in IMAGE_SHIFTS:
        shift = (C.c_double * 3)(*(float(v) * p["boxsize"] for v in s))
        lib.fmm_remote(0, shift)
    first_node = C.c_int.in_dll(lib, "first_node").value
    first_leaf, last_leaf = C.c_int.in_dll(lib, "first_leaf").value, C.c_int.in_dll(lib, "last_leaf").value
    lib.walk_l2l(first_node)
    for n in range(first_leaf, last_leaf):
        lib.l2p(n)
    assert rel_err(part["acc"], g["acc"], p).max() <= 1e-10
    c = ref.counters()
    assert [c[k] for k in ("idxP2P", "idxM2L", "walk_m2l_count", "p2p_count_remote")] == list(g["counters"][:4])
    ref.deconstruct()


@pytest.mark.parametrize("entry", ["p2p_kernel", "p2p_kernel_rinvsqrt"])
def test_kernels_h_leaf_pairs_sum_to_the_local_task_phase(ph, entry):
    """The inc/kernels.h entry points, one call per task of the reference's
    own local P2P list (in its order; a leaf with itself through
    p2p_kernel_inleaf), after fmm_prepare: part[].acc equals the
    reference's accelerations after fmm_task (no M2L in this fixture)."""
    g = load_golden("grid16_leaf16")
    p = g["p"]
    ref = ph.Reference()
    ref.setup(g["pos_in"], p)
    lib = ref.lib
    for name in ("p2p_kernel", "p2p_kernel_rinvsqrt", "p2p_kernel_inleaf"):
        getattr(lib, name).argtypes = [C_int(), C_int()]
        getattr(lib, name).restype = None
    lib.fmm_construct()
    lib.fmm_prepare()
    part = ref.part()
    part["acc"] = 0.0
    fn = getattr(lib, entry)
    t, s, _ = g["list_p2p"]
    for a, b in zip(t.tolist(), s.tolist()):
        if a == b and entry == "p2p_kernel":
            lib.p2p_kernel_inleaf(a, b)
        else:
            fn(a, b)
    assert ph.load_library().photons_gpu_status() == 0
    assert rel_err(part["acc"], g["acc_task"], p).max() <= 1e-10
    ref.deconstruct()


def C_int():
    import ctypes
    return ctypes.c_int


@pytest.mark.parametrize("n,rmax,eps,reach", [
    (1, 3.0, 0.1, 1.0),      # no source but the target
    (33, 40.0, 0.1, 1.0),    # one cell: every source, nearest images
    (700, 2.0, 0.0, 1.0),    # five cells a side, unsoftened
    (700, 3.3, 0.5, 1.0),    # three cells a side, softening above the spacing
    (2000, 3.0, 0.1, 3.0),   # positions up to three sides from the origin (folded once)
    (2000, 0.5, 0.1, 1.0)])  # few sources within rmax
def test_direct_sum_filter_keeps_every_source(ph, n, rmax, eps, reach):
    """The direct sum against numpy: the FP32 distance filter in front of the
    exact test drops nothing within rmax.  Tolerance: 1e-13 of the sum of the
    contributions' magnitudes (a few hundred terms of a few ulp each)."""
    from scipy.special import erfc
    L, rs, m = 10.0, 0.6, 2.5
    rng = np.random.default_rng(n)
    pos = rng.uniform(0.0, L * reach, (n, 3)) if reach == 1.0 else rng.uniform(-L * reach, L * reach, (n, 3))
    targets = rng.choice(n, min(n, 40), replace=False).astype(np.int32)
    p = dict(boxsize=L, theta=0.5, rs=rs, rcut=4.5 * rs, eps=eps, mass=m, maxleaf=16)
    got = ph.direct_sum(pos, p, targets, rmax)
    ncell = int(L / rmax)
    ncell = 1 if ncell < 3 else min(ncell, 512)
    cell = np.clip((pos / (L / ncell)).astype(np.int64), 0, ncell - 1)
    for k, t in enumerate(targets):
        d = pos - pos[t]
        d = np.where(d > 0.5 * L, d - L, np.where(d < -0.5 * L, d + L, d))
        r = np.sqrt((d ** 2).sum(1))
        step = np.abs(cell - cell[t])
        near = (np.minimum(step, ncell - step) <= 1).all(1) if ncell >= 3 else np.ones(n, bool)
        on = near & (r < rmax) & (np.arange(n) != t)
        u = 0.5 * r[on] / rs
        f = m * (erfc(u) + 2.0 / np.sqrt(np.pi) * u * np.exp(-u * u)) / np.maximum(r[on], eps) ** 3
        want = (f[:, None] * d[on]).sum(0)
        scale = (np.abs(f)[:, None] * np.abs(d[on])).sum() + 1e-300
        assert np.abs(got[k] - want).max() <= 1e-13 * scale, (n, t)


def test_direct_sum_without_room_for_all_sources(ph, port, ics, monkeypatch):
    """With the buffer of the unbinned sum refused (the test hook), the call
    takes the binned sum: the bar of the direct sum above."""
    pos, p = ics.make("nfw128", nside=24)
    targets = np.random.default_rng(5).choice(pos.shape[0], 300, replace=False).astype(np.int32)
    monkeypatch.setenv("PHOTONS_TEST_DIRECT_NO_ROOM", "1")
    got = ph.direct_sum(pos, p, targets)
    assert rel_err(got, port.direct_sum(pos, p, targets, nthreads=8), p).max() <= 1e-10


@pytest.mark.parametrize("rs", [-0.7, -1e3, -1e-3])
def test_direct_sum_of_a_negative_split_scale(ph, rs):
    """The direct sum does not refuse rs < 0: the reference's expressions at
    u < 0, binned and not.  Tolerance: 1e-13 of the sum of the magnitudes."""
    from scipy.special import erfc
    L, m, eps, n = 10.0, 2.5, 0.05, 300
    rng = np.random.default_rng(2)
    p = dict(boxsize=L, theta=0.5, rs=rs, rcut=3.0, eps=eps, mass=m, maxleaf=16)
    for pos in (rng.uniform(0.0, L, (n, 3)), rng.uniform(-1.0, L, (n, 3))):
        targets = np.arange(0, n, 10, dtype=np.int32)
        got = ph.direct_sum(pos, p, targets, 2.0 * L)
        for k, t in enumerate(targets):
            d = pos - pos[t]
            d = np.where(d > 0.5 * L, d - L, np.where(d < -0.5 * L, d + L, d))
            r = np.sqrt((d ** 2).sum(1))
            on = np.arange(n) != t
            u = 0.5 * r[on] / rs
            with np.errstate(over="ignore"):
                f = m * (erfc(u) + 2.0 / np.sqrt(np.pi) * u * np.exp(-u * u)) / np.maximum(r[on], eps) ** 3
            assert np.abs(got[k] - (f[:, None] * d[on]).sum(0)).max() <= 1e-13 * (np.abs(f) * r[on]).sum()


@pytest.mark.parametrize("rs", [1e-160, 1e-3, 0.7, 1e3, 1e50, 1e100, 1e160, np.inf])
def test_fp64_forces_at_extreme_split_scales(ph, rs):
    """From no long-range part at all (rs far above the box: Newtonian forces)
    to nothing but it (rs far below the spacing: none): the FP64 pass, mutual
    and one way, and the direct sum against numpy.  Tolerance: as above."""
    from scipy.special import erfc
    L, m, eps, n = 10.0, 2.5, 0.05, 400
    pos = np.random.default_rng(1).uniform(0.0, L, (n, 3))
    targets = np.arange(0, n, 10, dtype=np.int32)
    # theta 0, a cutoff beyond the images: all 27 images of every pair
    p = dict(boxsize=L, theta=0.0, rs=rs, rcut=4.0 * L, eps=eps, mass=m, maxleaf=8)

    def check(got, near):
        for k, t in enumerate(targets):
            want, scale = np.zeros(3), 1e-300
            d = pos - pos[t]
            shifts = [(0, 0, 0)] if near else [(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)]
            for sh in shifts:
                e = d - L * np.round(d / L) if near else d + L * np.array(sh)
                r = np.sqrt((e ** 2).sum(1))
                on = r > 0
                u = 0.5 * r[on] / rs
                f = m * (erfc(u) + 2.0 / np.sqrt(np.pi) * u * np.exp(-np.minimum(u, 1e3) ** 2)) / np.maximum(r[on], eps) ** 3
                want += (f[:, None] * e[on]).sum(0)
                scale += (f * r[on]).sum()
            assert np.abs(got[k] - want).max() <= 1e-13 * scale

    with contextlib.closing(ph.ForcePass(0)) as fp:
        for flags in (0, ph.F_ONE_WAY):
            check(fp.run(pos, p, precision=ph.FP64, flags=flags)[targets], False)
    check(ph.direct_sum(pos, p, targets, 2.0 * L), True)


@pytest.mark.parametrize("ntarget", [1, 9, 4096, 4097])
def test_direct_sum_slices_and_bins_match_oracle(ph, port, ics, ntarget):
    """The direct sum with the sources in several slices (few targets) and
    over binned sources (more than 4,096): the bar of the direct sum above."""
    pos, p = ics.make("nfw128", nside=32)
    targets = np.random.default_rng(5).choice(pos.shape[0], ntarget, replace=False).astype(np.int32)
    got = ph.direct_sum(pos, p, targets)
    want = port.direct_sum(pos, p, targets, nthreads=8)
    assert rel_err(got, want, p).max() <= 1e-10


@pytest.mark.parametrize("nside,L", [(4, 1.0), (37, 10.0), (64, 64.0), (64, 3.0e-7), (50, 1.0e9)])
def test_pm_weights_at_cell_edges_match_oracle(ph, nside, L):
    """The PM where the integer weights meet their edges: positions at cell
    boundaries and centres, the box's two faces, just below zero, one last
    place to either side, tiny ones, and random ones.  The bar of the golden
    PM test."""
    import pm_oracle
    rng = np.random.default_rng(nside)
    h = L / nside
    edge = np.concatenate([np.arange(nside + 1) * h, (np.arange(nside) + 0.5) * h])
    edge = np.concatenate([edge, np.nextafter(edge, 0.0), np.nextafter(edge, 2 * L),
                           [0.0, -0.0, -0.25 * h, -1e-9 * h, 1e-300, 1e-20 * L, L]])
    pos = np.concatenate([rng.choice(edge, (400, 3)), rng.uniform(0.0, L, (400, 3)),
                          np.mod(rng.normal(0.3 * L, 0.01 * L, (400, 3)), L)])
    p = dict(boxsize=L, theta=0.5, rs=1.25 * h, rcut=6.0 * h, eps=0.0, mass=2.5, maxleaf=16)
    with contextlib.closing(ph.ForcePass(0)) as fp:
        got = fp.pm_force(pos, p, nside)
    want = pm_oracle.pm_force(pos, L, nside, p["rs"], p["mass"])
    assert np.abs(got - want).max() <= 1e-10 * np.abs(want).max()


@pytest.mark.parametrize("nside,L", [(5, 1.0), (37, 10.0), (64, 3.0e-7)])
def test_pm_of_positions_below_the_box_matches_oracle(ph, nside, L):
    """Positions up to 2.9 cells below the box, where the reference's
    truncated cell index gives weights between -0.5 and 1.5: the bar above."""
    import pm_oracle
    rng = np.random.default_rng(nside)
    h = L / nside
    below = np.concatenate([[-0.75 * h, -1.6 * h, -0.5 * h, -1.5 * h, -h, np.nextafter(-0.5 * h, -L)],
                            rng.uniform(-2.9 * h, 0.0, 200)])
    pos = np.concatenate([rng.choice(below, (300, 3)), rng.uniform(0.0, L, (300, 3))])
    pos[300:500, 1] = rng.choice(below, 200)
    p = dict(boxsize=L, theta=0.5, rs=1.25 * h, rcut=6.0 * h, eps=0.0, mass=2.5, maxleaf=16)
    with contextlib.closing(ph.ForcePass(0)) as fp:
        got = fp.pm_force(pos, p, nside)
    want = pm_oracle.pm_force(pos, L, nside, p["rs"], p["mass"])
    assert np.abs(got - want).max() <= 1e-10 * np.abs(want).max()


@pytest.mark.parametrize("workload,n,nside", [("grid32", 24, 32), ("nfw128", 28, 40), ("zeldovich256", 24, 24)])
def test_pm_is_as_accurate_as_an_fp64_evaluation(ph, ics, workload, n, nside):
    """The 64-bit integer PM and the FP64 oracle, both against extended
    precision: at most twice the oracle's rms error (their transforms round
    differently; the terms the integers replace are a small part of it)."""
    import pm_oracle
    pos, p = ics.make(workload, nside=n)
    args = (pos, p["boxsize"], nside, p["rs"], p["mass"])
    want = pm_oracle.pm_force(*args, real=np.longdouble)
    assert want.dtype == np.longdouble
    with contextlib.closing(ph.ForcePass(0)) as fp:
        got = fp.pm_force(pos, p, nside)
    rms = lambda x: float(np.sqrt(((x - want) ** 2).mean()))  # noqa: E731
    assert rms(got) <= 2.0 * rms(pm_oracle.pm_force(*args)), (rms(got), rms(pm_oracle.pm_force(*args)))


def test_pm_of_a_position_that_is_not_finite_is_nan(ph):
    pos = np.random.default_rng(0).uniform(0.0, 8.0, (50, 3))
    pos[7, 1] = np.nan
    p = dict(boxsize=8.0, theta=0.5, rs=1.0, rcut=4.0, eps=0.0, mass=1.0, maxleaf=16)
    with contextlib.closing(ph.ForcePass(0)) as fp:
        assert np.isnan(fp.pm_force(pos, p, 8)).all()
