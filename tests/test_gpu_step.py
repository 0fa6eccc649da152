"""GPU parity of the full liquid substep (sort -> P2G + normalize + gravity ->
MGPCG projection -> G2P + advection) against the FP64 oracle on the seeded dam
break, at 32^3 (steps 1 and 10, oracle replayed from the GPU state) and 128^3.

Tolerances: grid and particle fields 1e-5 norm-wise relative (FP32 transfers
vs FP64 oracle); pressure 1e-5 relative (both solves stop at a 1e-6 relative
FP64 residual); the GPU pressure's own FP64 residual, re-evaluated by the
oracle, <= 1e-6 ||b||."""

import ctypes

import numpy as np
import pytest

import fluidity_b200 as fb
import oracle
from fluidity_b200 import scenes
from helpers import box_for, dam_break_context, read_fields, rel_err, soa_to_xvc, sort_permutation
from oracle.box_system import box_pressure_system

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _compare_step(ctx, n, state_in, precision=0, levels=0, pre=1, post=2):
    """Runs one GPU step from state_in and one oracle step; returns errors."""
    ctx.upload(state_in)
    code, diag = ctx.step(fb.transfer_params(scenes.DT, scenes.DENSITY / n ** 3 / 8),
                          fb.default_pressure_options(precision=precision, levels=levels, pre=pre, post=post))
    assert code == fb.OK, diag.as_dict()
    f = read_fields(ctx, n)
    out = ctx.download()
    x, v, c = soa_to_xvc(state_in)
    box = box_for(n)
    r = oracle.step(box, x, v, c, scenes.DT)
    perm = sort_permutation(state_in, n)
    errs = {}
    for a in range(3):
        have = ~np.isnan(f["u_pred"][a])
        errs[f"u_pred{a}"] = rel_err(f["u_pred"][a], r["u_pred"][a], have)
        errs[f"u_new{a}"] = rel_err(f["u_new"][a], r["u_new"][a], have)
    fluid = r["cell_type"] == 1
    known = f["cell_type"] != 255
    assert np.array_equal(f["cell_type"][known], r["cell_type"][known])
    assert not np.any(fluid & ~known)
    errs["pressure"] = rel_err(f["pressure"], r["pressure"], fluid)
    errs["x"] = float(np.abs(out[0:3].T - r["x"][perm]).max() / n)  # in cells
    errs["v"] = rel_err(out[3:6].T, r["v"][perm])
    errs["C"] = rel_err(out[6:15].T, r["c"][perm])
    return errs, diag, f, out


@pytest.mark.parametrize("precision", [0, 1])
def test_dam_break_32_first_step_matches_oracle(precision):
    ctx, soa, _ = dam_break_context(32)
    errs, diag, _, _ = _compare_step(ctx, 32, soa, precision)
    assert diag.relative_residual <= 1e-6
    for k, e in errs.items():
        assert e <= TOL, (k, e, errs)


def test_dam_break_32_step_10_matches_oracle_replay():
    ctx, soa, m = dam_break_context(32)
    tp = fb.transfer_params(scenes.DT, m)
    opt = fb.default_pressure_options()
    for _ in range(9):
        code, _ = ctx.step(tp, opt)
        assert code == fb.OK
    state9 = ctx.download()
    errs, diag, _, _ = _compare_step(ctx, 32, state9)
    for k, e in errs.items():
        assert e <= TOL, (k, e, errs)


def test_dam_break_32_step_100_matches_oracle_replay():
    """Config 1 runs 100 steps: the 100th step, replayed by the oracle from the GPU state."""
    ctx, soa, m = dam_break_context(32)
    tp = fb.transfer_params(scenes.DT, m)
    opt = fb.default_pressure_options()
    for _ in range(99):
        code, _ = ctx.step(tp, opt)
        assert code == fb.OK
    errs, diag, _, _ = _compare_step(ctx, 32, ctx.download())
    assert diag.relative_residual <= 1e-6
    for k, e in errs.items():
        assert e <= TOL, (k, e, errs)


def test_dam_break_128_steps_10_and_200_match_oracle_replay():
    """Config 2 (128^3, 4-level V-cycle): steps 10 and 200, each replayed by the
    oracle from the GPU state of the step before."""
    ctx, soa, m = dam_break_context(128)
    tp = fb.transfer_params(scenes.DT, m)
    opt = fb.default_pressure_options(levels=4, pre=2, post=2)
    done = 0
    for check in (10, 200):
        while done < check - 1:
            code, _ = ctx.step(tp, opt)
            assert code == fb.OK
            done += 1
        errs, diag, _, _ = _compare_step(ctx, 128, ctx.download(), levels=4, pre=2, post=2)
        done += 1
        assert diag.relative_residual <= 1e-6
        for k, e in errs.items():
            assert e <= TOL, (check, k, e, errs)


def test_dam_break_128_first_step_matches_oracle():
    """128^3 with the 4-level V-cycle (2 pre + 2 post red-black sweeps)."""
    ctx, soa, _ = dam_break_context(128)
    errs, diag, _, _ = _compare_step(ctx, 128, soa, levels=4, pre=2, post=2)
    assert diag.levels == 4
    for k, e in errs.items():
        assert e <= TOL, (k, e, errs)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("warm_start", [0, 2])
def test_pressure_meets_fp64_residual_checked_by_oracle(precision, warm_start):
    """The GPU pressure, re-evaluated in FP64 by the oracle on the same system
    (built from the GPU's own predicted velocities), meets 1e-6 ||b||, and the
    reference's own gate is reported; from p = 0 and from the pressure
    extrapolated from the last two projections."""
    n = 64
    ctx, soa, m = dam_break_context(n)
    opt = fb.default_pressure_options(precision=precision, warm_start=warm_start)
    for _ in range(3):
        ctx.step(fb.transfer_params(scenes.DT, m), opt)
    code, diag = ctx.step(fb.transfer_params(scenes.DT, m), opt)
    assert code == fb.OK
    f = read_fields(ctx, n)
    box = box_for(n)
    u_pred = [np.nan_to_num(f["u_pred"][a].astype(np.float64)) for a in range(3)]
    ct = np.where(f["cell_type"] == 255, 2, f["cell_type"]).astype(np.uint8)
    sysm = box_pressure_system(box, ct, u_pred)
    ci = sysm["cells_idx"]
    p = f["pressure"][ci[:, 2], ci[:, 1], ci[:, 0]]
    ev = oracle.pressure_evaluate(sysm["cells_idx"], sysm["cells_val"], sysm["faces_idx"], sysm["faces_kind"],
                                  sysm["faces_val"], box.h, scenes.DT, p)
    assert ev["diag"]["true_residual_l2"] <= 1.0001e-6 * ev["diag"]["rhs_l2"]
    assert diag.true_residual_l2 == pytest.approx(ev["diag"]["true_residual_l2"], rel=1e-3)
    assert diag.true_residual_l2 <= diag.reference_limit


def test_step_is_bitwise_reproducible():
    ctx, soa, m = dam_break_context(32)
    tp, opt = fb.transfer_params(scenes.DT, m), fb.default_pressure_options()
    outs = []
    for _ in range(2):
        ctx.upload(soa)
        for _ in range(3):
            ctx.step(tp, opt)
        f = read_fields(ctx, 32)
        outs.append((ctx.download(), f["u_new"], f["pressure"]))
    np.testing.assert_array_equal(outs[0][0], outs[1][0])
    for a in range(3):
        np.testing.assert_array_equal(outs[0][1][a], outs[1][1][a])
    np.testing.assert_array_equal(outs[0][2], outs[1][2])


@pytest.mark.parametrize("precision,tol", [(0, 1e-5), (1, 3e-2)])
@pytest.mark.parametrize("n,levels", [(32, 4), (64, 5)])
def test_vcycle_matches_fp64_restatement(precision, tol, n, levels):
    """One V-cycle against the FP64 restatement. At 64^3 with 5 levels the last
    dense level (8^3) and the coarsest (4^3) run in the one-CTA coarse tail."""
    ctx, soa, m = dam_break_context(n)
    ctx.step(fb.transfer_params(scenes.DT, m), fb.default_pressure_options())
    blocks = ctx.active_blocks()
    nb = len(blocks)
    f = read_fields(ctx, n)
    ct = np.where(f["cell_type"] == 255, 2, f["cell_type"]).astype(np.uint8)
    rng = np.random.default_rng(7)
    r_dense = rng.normal(size=ct.shape) * (ct == 1)
    # dense -> sparse layout
    loc = np.arange(512)
    gx = (blocks[:, 0:1] * 8 + (loc & 7)).ravel()
    gy = (blocks[:, 1:2] * 8 + ((loc >> 3) & 7)).ravel()
    gz = (blocks[:, 2:3] * 8 + (loc >> 6)).ravel()
    r_sparse = r_dense[gz, gy, gx].astype(np.float32)
    lib = fb.library()
    import torch
    r_dev = torch.from_numpy(r_sparse).cuda()
    z_dev = torch.zeros_like(r_dev)
    opt = fb.default_pressure_options(precision=precision, levels=levels)
    assert lib.fl_apply_vcycle(ctx.handle, ctypes.c_void_p(r_dev.data_ptr()), ctypes.c_void_p(z_dev.data_ptr()),
                               ctypes.byref(opt), None) == fb.OK
    torch.cuda.synchronize()
    z = fb.sparse_cells_to_dense(blocks, z_dev.cpu().numpy(), (n, n, n))
    zo = oracle.vcycle(box_for(n), ct, r_dense, levels=levels, pre=opt.pre_sweeps, post=opt.post_sweeps,
                       coarse_sweeps=opt.coarse_sweeps)
    assert rel_err(z, zo, ct == 1) <= tol


def test_sort_is_a_stable_cell_permutation():
    n = 32
    ctx, soa, m = dam_break_context(n)
    rng = np.random.default_rng(3)
    shuffled = soa[:, rng.permutation(soa.shape[1])].copy()
    ctx.upload(shuffled)
    ctx.step(fb.transfer_params(0.0, m, gravity=(0, 0, 0)), fb.default_pressure_options())
    out = ctx.download()
    perm = sort_permutation(shuffled, n)
    # dt = 0: positions only move by the wall clamp (<= 1e-3 h); the order is the stable cell sort
    np.testing.assert_allclose(out[0:3], shuffled[0:3, perm], rtol=0, atol=1.01e-3 / n)
    f = ctx.fields()
    nb = len(ctx.active_blocks())
    cs = fb.copy_to_host(f["cell_start"], nb * 512 + 1, np.int32)
    assert cs[0] == 0 and cs[-1] == soa.shape[1] and np.all(np.diff(cs) >= 0)


def test_sort_handles_crowded_blocks():
    """A block holding more particles than the sort stages in shared memory
    (12,288) sorts its cells in place; the order is still the stable cell sort,
    next to a block that takes the staged path."""
    n = 32
    rng = np.random.default_rng(5)
    crowded, normal = 20000, 3000
    x = np.concatenate([rng.uniform(8.0 / n, 16.0 / n, size=(3, crowded)),
                        rng.uniform([[16.0 / n], [8.0 / n], [8.0 / n]], [[24.0 / n], [16.0 / n], [16.0 / n]],
                                    size=(3, normal))], axis=1)
    soa = np.zeros((15, crowded + normal), np.float32)
    soa[0:3] = x[:, rng.permutation(x.shape[1])]
    soa[3:6] = rng.normal(scale=0.1, size=(3, soa.shape[1]))
    ctx = fb.LiquidContext(n, capacity=soa.shape[1])
    ctx.upload(soa)
    code, diag = ctx.step(fb.transfer_params(0.0, 1.0 / (8 * n ** 3), gravity=(0, 0, 0)),
                          fb.default_pressure_options())
    assert code == fb.OK
    out = ctx.download()
    perm = sort_permutation(soa, n)
    np.testing.assert_array_equal(out[0:3], soa[0:3, perm])  # dt = 0, far from the walls: x unchanged
    f = ctx.fields()
    nb = len(ctx.active_blocks())
    cs = fb.copy_to_host(f["cell_start"], nb * 512 + 1, np.int32)
    assert cs[0] == 0 and cs[-1] == soa.shape[1] and np.all(np.diff(cs) >= 0)
    ctx.close()


def test_empty_and_invalid_particles():
    ctx = fb.LiquidContext(32, capacity=64)
    ctx.upload(np.zeros((15, 0), np.float32))
    code, diag = ctx.step(fb.transfer_params(scenes.DT, 1.0), fb.default_pressure_options())
    assert code == fb.OK
    bad = np.zeros((15, 2), np.float32)
    bad[0:3] = 0.5
    bad[0, 1] = 2.0  # outside the box lattice
    ctx.upload(bad)
    with pytest.raises(fb.FluidityError) as e:
        ctx.step(fb.transfer_params(scenes.DT, 1.0), fb.default_pressure_options())
    assert e.value.code == fb.FAILED_PRECONDITION
    bad[0, 1] = np.nan
    ctx.upload(bad)
    with pytest.raises(fb.FluidityError) as e:
        ctx.step(fb.transfer_params(scenes.DT, 1.0), fb.default_pressure_options())
    assert e.value.code == fb.OUT_OF_RANGE
    with pytest.raises(fb.FluidityError) as e:
        ctx.upload(np.zeros((15, 65), np.float32))
    assert e.value.code == fb.RESOURCE_EXHAUSTED


def _in_runs(count, rng, n, run):
    """Positions whose blocks come in runs of `run` particles (0: in no order, some blocks with many).
    Runs beyond 12 are of the same 12 blocks, so that most blocks of the lattice stay empty, and six
    particles anywhere among them are alone in their blocks: each of those marks is made once."""
    if run == 0:
        x = rng.uniform(1.0 / n, 1.0 - 1.0 / n, size=(3, count))
        x[:, ::2] *= 0.25
        return x
    blocks = rng.permutation((n // 8) ** 3)
    of = np.repeat(np.resize(blocks[:12], -(-count // run)), run)[:count]
    if count > 1000:
        of[rng.choice(count, 6, replace=False)] = blocks[12:18]
    return (8 * np.stack([of % (n // 8), of // (n // 8) % (n // 8), of // (n // 8) ** 2]) +
            rng.uniform(0.01, 7.99, size=(3, count))) / n


@pytest.mark.parametrize("run", [0, 3, 4, 5, 31, 33, 128, 200])
@pytest.mark.parametrize("count", [1, 31, 33, 127, 129, 1023, 1024, 1025, 5000, 454656, 454657, 500003])
def test_topology_from_unordered_particles(count, run):
    """Blocks marked by particles in no order and in runs of a block (around the 8 runs a turn of 32
    and around a warp's 128 particles), at counts around a turn, a warp, the 1024 particles of a CTA and
    the 444 CTAs above which a CTA's blocks are joined before they are looked up, against the blocks
    (and their ring) found on the host; a particle that has no block is reported with its index."""
    import torch

    n, rng = 128, np.random.default_rng(count)
    soa = np.zeros((15, count), np.float32)
    soa[0:3] = _in_runs(count, rng, n, run)
    ctx = fb.LiquidContext(n, capacity=count)
    dev = torch.from_numpy(soa).cuda()
    p = fb.Particles()
    p.x[:] = [dev[d].data_ptr() for d in range(3)]
    p.v[:] = [dev[3 + d].data_ptr() for d in range(3)]
    p.c[:] = [dev[6 + d].data_ptr() for d in range(9)]
    p.mass, p.count = None, count
    lib, rep = fb.library(), fb.Report()
    assert lib.fl_topology_from_particles(ctx.handle, ctypes.byref(p), None, ctypes.byref(rep)) == fb.OK
    blk = np.floor(soa[0:3] * np.float32(n)).astype(int) // 8
    occ = np.zeros((18, 18, 18), bool)
    for dz in range(3):
        for dy in range(3):
            for dx in range(3):
                occ[blk[2] + dz, blk[1] + dy, blk[0] + dx] = True
    z, y, x = np.nonzero(occ[1:17, 1:17, 1:17])
    np.testing.assert_array_equal(ctx.active_blocks(), np.stack([x, y, z], 1))
    for bad, code in ((np.nan, fb.OUT_OF_RANGE), (1.5, fb.FAILED_PRECONDITION)):
        dev[1, count - 1] = bad
        assert lib.fl_topology_from_particles(ctx.handle, ctypes.byref(p), None, ctypes.byref(rep)) == code
        assert rep.first_bad_index == count - 1
    ctx.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [24, 144, 152])
def test_flexible_cg_scalars_by_block_count(precision, n):
    """The flexible-CG scalars are summed by the kernels that use them up to 1024 active blocks (24^3:
    27, 144^3: 1000) and by kernels of their own above (152^3: 1331). Both reach the 1e-6 FP64
    residual, and a second solve of the same system repeats the first's bits."""
    ctx, soa, m = dam_break_context(n)
    tp, opt = fb.transfer_params(scenes.DT, m), fb.default_pressure_options(precision=precision)
    code, diag = ctx.step(tp, opt)
    assert code == fb.OK and diag.relative_residual <= 1e-6
    assert (diag.active_blocks <= 1024) == (n < 150)
    runs = []
    for _ in range(2):
        code, d = ctx.project(tp, opt)
        assert code == fb.OK and d.relative_residual <= 1e-6 and d.iterations <= 20
        f = ctx.fields()
        runs.append(fb.copy_to_host(f["pressure"], d.active_blocks * 512, np.float64))
    np.testing.assert_array_equal(runs[0], runs[1])
    ctx.close()


@pytest.mark.parametrize("precision,tol", [(0, 1e-5), (1, 3e-2)])
@pytest.mark.parametrize("n,levels", [(24, 4), (40, 5), (72, 6), (176, 0)])
def test_vcycle_coarse_levels_in_a_cluster(precision, tol, n, levels):
    """One V-cycle against the FP64 restatement where the levels below level 0 or 1 run in one
    cluster: odd block lattices (3, 5, 9 and 22 blocks), fewer blocks than CTAs, the coarsest level
    right below the in-block ones (4 levels) and, at 176^3 in FP32, more blocks than level 1 may have."""
    import torch

    ctx, soa, m = dam_break_context(n)
    ctx.step(fb.transfer_params(scenes.DT, m), fb.default_pressure_options())
    blocks, f = ctx.active_blocks(), read_fields(ctx, n)
    ct = np.where(f["cell_type"] == 255, 2, f["cell_type"]).astype(np.uint8)
    r_dense = np.random.default_rng(n).normal(size=ct.shape) * (ct == 1)
    loc = np.arange(512)
    gx, gy, gz = ((blocks[:, d:d + 1] * 8 + (loc >> 3 * d & 7)).ravel() for d in range(3))
    r_dev = torch.from_numpy(r_dense[gz, gy, gx].astype(np.float32)).cuda()
    z_dev = torch.zeros_like(r_dev)
    opt = fb.default_pressure_options(precision=precision, levels=levels)
    assert fb.library().fl_apply_vcycle(ctx.handle, r_dev.data_ptr(), z_dev.data_ptr(), ctypes.byref(opt), None) == fb.OK
    torch.cuda.synchronize()
    if levels == 0:  # the library's rule: the first dense level of at most 512 cells is the coarsest
        levels = next(l for l in range(4, 12) if (-(-(n // 8) // 2 ** (l - 4))) ** 3 <= 512)
    z = fb.sparse_cells_to_dense(blocks, z_dev.cpu().numpy(), (n, n, n))
    zo = oracle.vcycle(box_for(n), ct, r_dense, levels=levels, pre=opt.pre_sweeps, post=opt.post_sweeps,
                       coarse_sweeps=opt.coarse_sweeps)
    assert rel_err(z, zo, ct == 1) <= tol
    ctx.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [24, 144, 152])
def test_solve_that_breaks_down_ends_and_leaves_no_trace(precision, n):
    """A predicted velocity that is not a number makes z.r not positive: the solve ends with ABORTED
    where the kernels that use the CG scalars sum them (27 and 1000 blocks) and where kernels of their
    own do (1331), after no iteration, and the next solve gives the bits of the one before."""
    import torch

    ctx, _, m = dam_break_context(n)
    tp, opt = fb.transfer_params(scenes.DT, m), fb.default_pressure_options(precision=precision)
    code, diag = ctx.step(tp, opt)
    assert code == fb.OK
    f, cells = ctx.fields(), diag.active_blocks * 512
    u = [torch.from_numpy(fb.copy_to_host(f["u_pred"][a], cells, np.float32)).cuda() for a in range(3)]
    out = [torch.zeros(cells, device="cuda") for _ in range(3)]
    arr = lambda ts: (ctypes.c_void_p * 3)(*[t.data_ptr() for t in ts])  # noqa: E731
    broken = [t.clone() for t in u]
    fluid = int(np.flatnonzero(fb.copy_to_host(f["cell_type"], cells, np.uint8) == 1)[-1])
    broken[1][fluid] = float("nan")
    p = torch.zeros(cells, dtype=torch.float64, device="cuda")
    pressures = []
    for velocities, want in ((u, fb.OK), (broken, fb.ABORTED), (u, fb.OK), (broken, fb.ABORTED), (u, fb.OK)):
        d = fb.PressureDiagnostics()
        code = fb.library().fl_pressure_project(ctx.handle, arr(velocities), arr(out), ctypes.byref(tp), ctypes.byref(opt),
                                                ctypes.byref(d), p.data_ptr(), None)
        assert code == want
        if code == fb.OK:
            pressures.append(p.cpu().numpy())
        else:
            assert d.status == fb.ABORTED and d.iterations == 0
    for other in pressures[1:]:
        np.testing.assert_array_equal(other, pressures[0])
    ctx.close()


def test_short_states_in_a_context_of_large_capacity():
    """Upload and download of a few particles where the arrays lie 2^31 bytes apart, more than
    the pitch that the device states for strided copies (76 GB of device memory, none of it touched beyond the particles)."""
    import torch

    if torch.cuda.mem_get_info()[0] < 90e9:
        pytest.skip("needs 90 GB of free device memory")
    rng = np.random.default_rng(8)
    soa = [rng.uniform(0.2, 0.8, size=(15, k)).astype(np.float32) for k in (1000, 7)]
    ctx = fb.LiquidContext(16, capacity=2 ** 29)
    for s in soa:
        ctx.upload(s)
        np.testing.assert_array_equal(ctx.download(), s)
    ctx.close()


@pytest.mark.parametrize("per", [1, 31, 32, 33, 129])
@pytest.mark.parametrize("order", ["cells", "pairs", "reversed"])
def test_sort_of_runs_of_equal_cells(per, order):
    """Particles whose cells come in runs around a warp's 32 lanes and the 128 particles of its four
    turns (a cell after the other, two cells in turn, the cells backwards), with a last warp that is not
    full: the stable cell sort, and a particle without a cell in the middle of a run is reported."""
    import torch

    n, cells = 32, 37
    rng = np.random.default_rng(per)
    cell = np.repeat(np.arange(cells), per)
    if order == "pairs":
        cell = np.concatenate([cell[0::2], cell[1::2]]) if per == 1 else cell.reshape(cells, per)[:36].reshape(18, 2, per).transpose(
            0, 2, 1).ravel()
    elif order == "reversed":
        cell = cell[::-1]
    x = np.stack([8 + cell % 8, 8 + cell // 8, np.full_like(cell, 9)]) + rng.uniform(0.05, 0.95, size=(3, len(cell)))
    soa = np.zeros((15, len(cell)), np.float32)
    soa[0:3] = x / n
    soa[3] = np.arange(len(cell))
    src, dst = torch.from_numpy(soa).cuda(), torch.zeros(soa.shape, device="cuda")

    def parts(t):
        p = fb.Particles()
        p.x[:] = [t[d].data_ptr() for d in range(3)]
        p.v[:] = [t[3 + d].data_ptr() for d in range(3)]
        p.c[:] = [t[6 + d].data_ptr() for d in range(9)]
        p.mass, p.count = None, soa.shape[1]
        return p

    ctx, lib, rep = fb.LiquidContext(n, capacity=len(cell)), fb.library(), fb.Report()
    a, b = parts(src), parts(dst)
    assert lib.fl_topology_from_particles(ctx.handle, ctypes.byref(a), None, ctypes.byref(rep)) == fb.OK
    assert lib.fl_sort_particles_by_block(ctx.handle, ctypes.byref(a), ctypes.byref(b), None, ctypes.byref(rep)) == fb.OK
    np.testing.assert_array_equal(dst.cpu().numpy(), soa[:, sort_permutation(soa, n)])
    bad = len(cell) // 2
    src[0, bad] = float("nan")
    assert lib.fl_sort_particles_by_block(ctx.handle, ctypes.byref(a), ctypes.byref(b), None,
                                          ctypes.byref(rep)) == fb.OUT_OF_RANGE
    assert rep.first_bad_index == bad
    ctx.close()


def test_sort_gathers_only_particles_that_have_a_cell():
    """Particles without a cell leave the sort's index shorter than the particles: in a context whose
    index still holds a longer sort's entries, and in a fresh one, the rest arrives in order and nothing
    from past the input (here: the longer sort's particles, in the same tensor) reaches the output."""
    import torch

    n = 32
    rng = np.random.default_rng(21)
    for before in (0, 5000):
        ctx, lib, rep = fb.LiquidContext(n, capacity=5000), fb.library(), fb.Report()
        soa = np.zeros((15, 5000), np.float32)
        soa[0:3] = rng.uniform(0.2, 0.8, size=(3, 5000))
        soa[3], soa[3, 700:] = np.arange(5000), -1.0
        src = torch.from_numpy(soa).cuda()
        for count, bad in ((before, 0), (700, 5)):
            if count == 0:
                continue
            dst = torch.full((15, 5000), 7.0, device="cuda")
            views = []
            for t in (src, dst):
                p = fb.Particles()
                p.x[:] = [t[d].data_ptr() for d in range(3)]
                p.v[:] = [t[3 + d].data_ptr() for d in range(3)]
                p.c[:] = [t[6 + d].data_ptr() for d in range(9)]
                p.mass, p.count = None, count
                views.append(p)
            a, b = views
            assert lib.fl_topology_from_particles(ctx.handle, ctypes.byref(a), None, ctypes.byref(rep)) == fb.OK
            good = np.ones(count, bool)
            good[rng.choice(count, bad, replace=False)] = False
            src[1, torch.from_numpy(np.flatnonzero(~good)).cuda()] = float("nan")
            code = lib.fl_sort_particles_by_block(ctx.handle, ctypes.byref(a), ctypes.byref(b), None, ctypes.byref(rep))
            assert code == (fb.OUT_OF_RANGE if bad else fb.OK)
            kept = soa[:, :count][:, good]
            got = dst.cpu().numpy()
            np.testing.assert_array_equal(got[:, :count - bad], kept[:, sort_permutation(kept, n)])
            if bad:
                assert np.all(got[3, count - bad:count] >= 0.0) and np.all(got[:, count:] == 7.0)
        ctx.close()
