"""GPU parity of the reference-mirror entry points (C ABI) against the golden
vectors produced by the reference itself and against the oracle."""
import ctypes as C

import numpy as np
import pytest

from bd_aging_b200 import configs as CF
from bd_aging_b200 import lib as B
from oracle import oracle as O

pytestmark = pytest.mark.gpu
SYSTEMS = ("g1", "g2")


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda:0")


def host(t):
    import torch
    torch.cuda.synchronize()
    return t.cpu().numpy()


def params(golden, name):
    return B.Parametros.from_buffer_copy(golden[name + "_params"].tobytes())


def cells(p, sp, rr_d):
    import torch
    nc = p.ncell_big if sp == "b" else p.ncell_sml
    nt = p.ntags_big if sp == "b" else p.ntags_sml
    nocup = torch.zeros(nc ** 3, dtype=torch.int32, device="cuda:0")
    cell = torch.zeros(nc ** 3 * nt, dtype=torch.int32, device="cuda:0")
    B.cell_locate(sp, rr_d, nocup, cell, p)
    return nocup, cell


@pytest.mark.parametrize("name", SYSTEMS)
def test_cell_locate_bit_exact(golden, name):
    p = params(golden, name)
    for sp in "bs":
        nocup, cell = cells(p, sp, dev(golden[name + "_r" + sp]))
        np.testing.assert_array_equal(host(nocup), golden[name + "_nocup_" + sp])
        np.testing.assert_array_equal(host(cell), golden[name + "_cell_" + sp])


def forces_four_calls(p, rb, rs):
    import torch
    rb_d, rs_d = dev(rb), dev(rs)
    nob, cb = cells(p, "b", rb_d)
    nos, cs = cells(p, "s", rs_d)
    z = lambda n, k: torch.zeros((n, k) if k > 1 else n, dtype=torch.float32, device="cuda:0")
    ffb, ffs = z(len(rb), 3), z(len(rs), 3)
    vb, pb, vs, ps = z(len(rb), 1), z(len(rb), 1), z(len(rs), 1), z(len(rs), 1)
    B.get_forces_same("b", rb_d, ffb, vb, pb, nob, cb, p)
    B.get_forces_same("s", rs_d, ffs, vs, ps, nos, cs, p)
    B.get_forces_diff("b", "s", rb_d, ffb, rs_d, vb, pb, nos, cs, p)
    B.get_forces_diff("s", "b", rs_d, ffs, rb_d, vs, ps, nob, cb, p)
    return dict(ff_b=host(ffb), ff_s=host(ffs), vir_b=host(vb), vir_s=host(vs), pot_b=host(pb), pot_s=host(ps))


@pytest.mark.parametrize("name", SYSTEMS)
def test_forces_match_reference(golden, name):
    p = params(golden, name)
    out = forces_four_calls(p, golden[name + "_rb"], golden[name + "_rs"])
    for k, v in out.items():
        ref = golden[name + "_" + k]
        # same neighbour sets and sum order as the reference host code; the
        # pair arithmetic may be fused (FMA) on the device
        np.testing.assert_allclose(v, ref, rtol=2e-5, atol=2e-5 * np.abs(ref).max(), err_msg=k)


@pytest.mark.parametrize("nb,ns,ntags", [(1, 2, 8), (33, 31, 9), (700, 500, 16), (700, 500, 17), (700, 500, 40),
                                         (8200, 33000, 16), (131073, 40000, 16)])
def test_cell_sort_and_force_paths_match_the_oracle(nb, ns, ntags):
    """16, 32 and more slots per cell (sorted by 16 or 32 lanes or a thread), a
    warp, eight lanes or a thread per particle by their number: cell lists exact, forces
    within the rounding of a float sum in another order."""
    side = CF.side_from_phi(max(nb, 60), max(ns, 60), 0.45)
    pos = CF.lattice_config(nb, ns, side, 17)
    p = O.setup_params(side, nb, ns, float(CF.SIGMA_BIG), float(CF.SIGMA_SML), ntags=(ntags, ntags))
    pp = B.Parametros.from_buffer_copy(bytes(p))
    for sp, rr in (("b", pos[:nb]), ("s", pos[nb:])):
        nocup, cell = cells(pp, sp, dev(rr))
        ref = O.cell_locate(p, sp, rr)
        np.testing.assert_array_equal(host(nocup), ref[0])
        np.testing.assert_array_equal(host(cell), ref[1])
    out, ref = forces_four_calls(pp, pos[:nb], pos[nb:]), O.ref_forces(p, pos[:nb].copy(), pos[nb:].copy())
    for k, v in out.items():
        np.testing.assert_allclose(v, ref[k], rtol=2e-5, atol=2e-5 * np.abs(ref[k]).max(), err_msg=k)


def test_a_thread_per_particle_over_125_cells_matches_the_oracle():
    """The first size at which the calls over 125 cells take a thread per particle."""
    nb, ns = 655361, 4000
    side = CF.side_from_phi(nb, ns, 0.3)
    pos = CF.lattice_config(nb, ns, side, 29)
    p = O.setup_params(side, nb, ns, float(CF.SIGMA_BIG), float(CF.SIGMA_SML), ntags=(16, 16))
    pp = B.Parametros.from_buffer_copy(bytes(p))
    assert pp.nrange_bs == 2
    out, ref = forces_four_calls(pp, pos[:nb], pos[nb:]), O.ref_forces(p, pos[:nb].copy(), pos[nb:].copy())
    for k, v in out.items():
        np.testing.assert_allclose(v, ref[k], rtol=2e-5, atol=2e-5 * np.abs(ref[k]).max(), err_msg=k)


@pytest.mark.parametrize("per_side,ntags", [(40, 16), (41, 16), (32, 17), (33, 17), (32, 32), (33, 32)])
def test_cell_lists_on_both_sides_of_the_lane_limit(per_side, ntags):
    """2^20 lanes in all (16 per cell, or 32 with more slots): cells sorted by
    lanes up to there, by a thread each beyond, unused slots -1 either way."""
    ss = float(CF.SIGMA_SML)
    side = float(np.float32((per_side + 0.5) * 1.05 * ss))
    n = 9000
    pos = np.random.default_rng(per_side + ntags).uniform(0, side, (n, 3)).astype(np.float32)
    pos[: ntags - 1] = np.float32(0.3) + pos[: ntags - 1] / np.float32(side)  # one nearly full cell
    p = O.setup_params(side, 10, n, float(CF.SIGMA_BIG), ss, ntags=(ntags, ntags))
    pp = B.Parametros.from_buffer_copy(bytes(p))
    assert pp.ncell_sml == per_side
    nocup, cell = cells(pp, "s", dev(pos))
    ref = O.cell_locate(p, "s", pos)
    np.testing.assert_array_equal(host(nocup), ref[0])
    np.testing.assert_array_equal(host(cell), ref[1])


@pytest.mark.parametrize("nb,ns", [(1000, 1200), (8200, 9000)])
def test_forces_of_a_drop_match_the_oracle(nb, ns):
    """A dense drop in an empty box: the lanes of a particle (32, then eight)
    visit full, half-full and empty cells, so they leave the cell loop at
    different times, and their sums still meet.  Same bounds as above."""
    inner = CF.side_from_phi(nb, ns, 0.5)
    side = float(np.float32(1.6 * inner))
    pos = (CF.lattice_config(nb, ns, inner, 23) + np.float32(0.2 * inner)).astype(np.float32)
    p = O.setup_params(side, nb, ns, float(CF.SIGMA_BIG), float(CF.SIGMA_SML), ntags=(16, 16))
    pp = B.Parametros.from_buffer_copy(bytes(p))
    out, ref = forces_four_calls(pp, pos[:nb], pos[nb:]), O.ref_forces(p, pos[:nb].copy(), pos[nb:].copy())
    for k, v in out.items():
        np.testing.assert_allclose(v, ref[k], rtol=2e-5, atol=2e-5 * np.abs(ref[k]).max(), err_msg=k)


@pytest.mark.parametrize("name", SYSTEMS)
def test_update_noise_bit_exact(golden, name):
    p = params(golden, name)
    for sp in "bs":
        rr = dev(golden[name + "_r" + sp])
        raw = rr.clone()
        B.update_ermak_noise(sp, rr, raw, dev(golden[name + "_ff_" + sp]), dev(golden[name + "_noise_" + sp]), p)
        np.testing.assert_array_equal(host(rr), golden[name + "_upd_rr_" + sp])
        np.testing.assert_array_equal(host(raw), golden[name + "_upd_raw_" + sp])


@pytest.mark.parametrize("name", SYSTEMS)
def test_gder_counts_exact(golden, name):
    import torch
    p = params(golden, name)
    rb, rs = dev(golden[name + "_rb"]), dev(golden[name + "_rs"])
    for pair, (a, b, ra, rbb) in zip(("bb", "bs", "sb", "ss"), (("b", "b", rb, rb), ("b", "s", rb, rs),
                                                               ("s", "b", rs, rb), ("s", "s", rs, rs))):
        counts = torch.zeros(p.nbins_gder, dtype=torch.int64, device="cuda:0")
        B.get_gder(a, b, ra, rbb, counts, p)
        np.testing.assert_array_equal(host(counts).astype(np.float64), golden[name + "_gder_" + pair], err_msg=pair)


def test_gder_counts_exact_larger_system():
    import torch
    nb = ns = 2000
    side = CF.side_from_phi(nb, ns, 0.5)
    pos = CF.lattice_config(nb, ns, side, 5)
    p = O.setup_params(side, nb, ns, float(CF.SIGMA_BIG), float(CF.SIGMA_SML), nbins=300, rng=side / 2)
    ref = O.gder_counts(p, pos[:nb], pos[nb:])
    pp = B.Parametros.from_buffer_copy(bytes(p))
    rb, rs = dev(pos[:nb]), dev(pos[nb:])
    for k, (a, b, ra, rbb) in enumerate((("b", "b", rb, rb), ("b", "s", rb, rs), ("s", "b", rs, rb),
                                         ("s", "s", rs, rs))):
        counts = torch.zeros(300, dtype=torch.int64, device="cuda:0")
        B.get_gder(a, b, ra, rbb, counts, pp)
        np.testing.assert_array_equal(host(counts).astype(np.uint64), ref[k])


@pytest.mark.parametrize("nb,ns,nbins,reach,where", [
    (1, 1, 7, 0.5, "fluid"), (255, 257, 200, 0.5, "fluid"), (256, 65, 8192, 0.49, "fluid"),
    (513, 511, 1, 0.87, "fluid"), (700, 343, 64, 0.8, "lattice"), (512, 512, 300, 0.5, "lattice"),
    (300, 200, 90, 0.6, "outside")])
def test_gder_counts_exact_edges(nb, ns, nbins, reach, where):
    """Sizes around a block of particles and a partner tile, one bin and the
    most bins, ranges below, at and beyond L / 2, a lattice whose separations
    are exact fractions of L (ties of the minimum image, distances on bin
    edges, coincident points), and coordinates outside the box."""
    import torch
    rng = np.random.default_rng(nb + nbins)
    side = 8.0 if where == "lattice" else CF.side_from_phi(nb + 60, ns + 60, 0.4)
    n = nb + ns
    if where == "lattice":
        pos = rng.integers(0, 9, (n, 3)).astype(np.float32)
    else:
        pos = rng.uniform(0, side, (n, 3)).astype(np.float32)
    if where == "outside":
        pos[::7] += np.float32(1.5 * side)
        pos[::11, 0] -= np.float32(3 * side)
    p = O.setup_params(side, nb, ns, float(CF.SIGMA_BIG), float(CF.SIGMA_SML), nbins=nbins, rng=reach * side)
    ref = O.gder_counts(p, pos[:nb].copy(), pos[nb:].copy())
    pp = B.Parametros.from_buffer_copy(bytes(p))
    rb, rs = dev(pos[:nb]), dev(pos[nb:])
    for k, (a, b, ra, rbb) in enumerate((("b", "b", rb, rb), ("b", "s", rb, rs), ("s", "b", rs, rb),
                                         ("s", "s", rs, rs))):
        counts = torch.zeros(nbins, dtype=torch.int64, device="cuda:0")
        B.get_gder(a, b, ra, rbb, counts, pp)
        np.testing.assert_array_equal(host(counts).astype(np.uint64), ref[k], err_msg=a + b)


def test_fself_and_msd(golden):
    raw, r0 = golden["g1_fself_raw_b"], golden["g1_rb"]
    fs = np.zeros(4, np.float32)
    B.fself_isotropic(dev(raw), dev(r0), len(r0), fs, 2, np.float32(7.0))
    np.testing.assert_allclose(fs, golden["g1_fself"], rtol=2e-6, atol=2e-7)
    m = B.msd(dev(raw), dev(r0), len(r0))
    assert abs(m - O.oracle_lib().or_ref_msd(raw, r0, len(r0))) < 1e-5 * m


def test_cell_overflow_is_reported_not_written_out_of_bounds():
    import torch
    nb, ns = 64, 64
    side = CF.side_from_phi(nb, ns, 0.3)
    p = B.setup_params(side, nb, ns, float(CF.SIGMA_BIG), float(CF.SIGMA_SML), ntags_big=2, ntags_sml=2)
    rr = np.full((nb, 3), 0.1, np.float32)  # every big particle in cell 0
    nocup = torch.zeros(p.ncell_big ** 3, dtype=torch.int32, device="cuda:0")
    guard = torch.full((p.ncell_big ** 3 * 2 + 64,), -7, dtype=torch.int32, device="cuda:0")
    cell = guard[: p.ncell_big ** 3 * 2]
    with pytest.raises(B.BDError) as ei:
        B.cell_locate("b", dev(rr), nocup, cell, p)
    assert ei.value.code == 3
    assert (host(guard)[p.ncell_big ** 3 * 2:] == -7).all()


def test_errors_of_many_particles_cost_no_more_than_one():
    """Every particle of a call can fail (outside the box, non-finite, a cell too
    full): each call reports its own error, a good one after it none, and a
    million failing particles take milliseconds at most."""
    import time
    n = 1 << 20
    side = CF.side_from_phi(n, n, 0.3)
    p = B.setup_params(side, n, n, float(CF.SIGMA_BIG), float(CF.SIGMA_SML))
    good = dev(np.random.default_rng(1).uniform(0, 0.9 * side, (n, 3)).astype(np.float32))
    few = B.setup_params(side, 1000, 1000, float(CF.SIGMA_BIG), float(CF.SIGMA_SML))
    for _ in range(2):
        for rr, code in ((good + 3 * side, 3), (good * float("nan"), 9), (good * 0 + 0.2, 3)):
            best = 1.0
            for _ in range(3):
                t = time.perf_counter()
                with pytest.raises(B.BDError) as ei:
                    cells(p, "b", rr)
                best = min(best, time.perf_counter() - t)
                assert ei.value.code == code
            assert best < 0.015
            cells(few, "b", good[:1000].clone())
        with pytest.raises(B.BDError) as ei:  # outside the box, each in a cell of its own
            cells(few, "b", good[:1000] + side)
        assert ei.value.code in (3, 1)


def test_two_contexts_keep_their_own_workspaces():
    """Calls that alternate between the primary context and another one of the
    same device give the same sums and allocate once per context."""
    n = 3000
    raw, r0 = np.random.default_rng(2).normal(size=(2, n, 3)).astype(np.float32)
    here = dev(raw), dev(r0)
    want = B.msd(*here, n)
    cu = C.CDLL("libcuda.so.1")

    def ok(rc):
        assert rc == 0, rc

    primary, other, free, total = C.c_void_p(), C.c_void_p(), C.c_size_t(), C.c_size_t()
    ok(cu.cuCtxGetCurrent(C.byref(primary)))
    ok(cu.cuCtxCreate_v2(C.byref(other), C.c_uint(0), C.c_int(0)))
    try:
        there = []
        for a in (raw, r0):
            p = C.c_uint64()
            ok(cu.cuMemAlloc_v2(C.byref(p), C.c_size_t(a.nbytes)))
            ok(cu.cuMemcpyHtoD_v2(p, C.c_void_p(a.ctypes.data), C.c_size_t(a.nbytes)))
            there.append(C.c_void_p(p.value))
        out = np.zeros(1, np.float32)
        level = []
        for _ in range(40):
            ok(cu.cuCtxSetCurrent(other))
            assert B.lib().bd_msd(there[0], there[1], n, C.c_void_p(out.ctypes.data), None) == 0
            assert out[0] == np.float32(want)
            ok(cu.cuMemGetInfo_v2(C.byref(free), C.byref(total)))
            level.append(free.value)
            ok(cu.cuCtxSetCurrent(primary))
            assert B.msd(*here, n) == want
        assert level[2] - level[-1] < 4 << 20
    finally:
        ok(cu.cuCtxSetCurrent(primary))
        ok(cu.cuCtxDestroy_v2(other))
    assert B.msd(*here, n) == want


def test_a_call_that_fails_waits_for_its_kernels():
    """An error left pending by the caller makes a call return after its launch;
    the workspace goes back only when that kernel is done, so the next call's
    result is its own."""
    import torch
    n = 100_000_000
    a = torch.ones((n, 3), device="cuda:0")
    b = torch.zeros((n, 3), device="cuda:0")
    want = B.msd(a[:1000], b[:1000], 1000)
    B.msd(a, b, n)
    torch.cuda.synchronize()
    rt = C.CDLL("libcudart.so.12")
    p = C.c_void_p()
    assert rt.cudaMalloc(C.byref(p), C.c_size_t(1 << 60)) != 0
    try:
        with pytest.raises(B.BDError):
            B.msd(a, b, n)  # about 0.4 ms of work
        idle = torch.cuda.default_stream().query()
    finally:
        rt.cudaGetLastError()
    assert idle
    assert B.msd(a[:1000], b[:1000], 1000) == want


def test_invalid_species_rejected():
    p = B.setup_params(10.0, 10, 10, 1.5, 1.1)
    with pytest.raises(B.BDError):
        B.cell_locate("x", None, None, None, p)
