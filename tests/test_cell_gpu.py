"""GPU parity, against the FP64 oracle, of the paths chosen by tracer count and
level count: stages as passes over cells (few tracers, the limited last stage
with tracers of both modes in a quad), the narrow form of the tiled stage (up
to 16 tracers), the grouped per-call step, and the acoustic step's kernels at
the level counts where a lane's or a column's share changes (32, 33, 64, 65
levels).

Tolerances are the repository's: 1e-5 normwise for the transport and the
thermodynamic fields, five times the oracle's own FP32-FP64 spread (at least
1e-5) for the momentum fields."""
import ctypes

import numpy as np
import pytest

import oracle_lib
from conftest import relerr, small_case
from olam_b200 import abi
from olam_b200.lib import HostState, OlamGpu
from test_dynamics_gpu import check_fields, dyn_case, gpu_long_steps, oracle_long_steps

pytestmark = pytest.mark.gpu

TOL = 1e-5


def case(nlev, ntr, w_amp, terrain):
    g, st = small_case(nxp=5, nlev=nlev, ntr=ntr, w_amp=w_amp, seed=23)
    if terrain:
        from olam_b200.synth.grid import with_terrain
        g = with_terrain(g, terrain)
    return g, st


def run(g, st, opts, pdef=None, coherence=abi.RESIDENT, steps=1, shape=None):
    dev = OlamGpu(abi.FortranGrid(g), opts, HostState(vmasc=st.vmasc, wmasc=st.wmasc, rho=st.rho, wc=st.wc))
    try:
        dev.set_coherence(coherence)
        rng = np.random.default_rng(3)
        var_p = [t.copy() for t in st.tracers]
        var_t = [(1e-6 * t * rng.standard_normal((t.shape[0], 1))).astype(np.float32) for t in st.tracers]
        sct = [t.copy() for t in var_t]
        dev.register_scalars(var_p, var_t, pdef=pdef)
        if shape:
            dev.set_tile_shape(*shape)
        for _ in range(steps):
            dev.scalar_transport_rk(st.rho_old)
        if coherence == abi.RESIDENT:
            dev.sync_to_host(abi.F_SCALARS)
        return np.stack(var_p), sct
    finally:
        dev.close()


def check(out, ref):
    for n in range(len(ref)):
        assert relerr(out[n][1:], ref[n][1:]) < TOL, (n, relerr(out[n][1:], ref[n][1:]))


# one tracer, a whole quad, a quad and one, the last counts of the cell passes
# and the first and last of the narrow tiles; levels below, at and above a
# warp's 32; w_amp 3: vertical CFL above 1, so implicit columns
@pytest.mark.parametrize("ntr,nlev,order,nrk,w_amp,terrain", [
    (1, 12, 2, 2, 0.05, 0), (1, 31, 3, 3, 3.0, 0), (4, 32, 2, 3, 0.05, 3), (5, 33, 3, 2, 0.05, 3),
    (8, 12, 2, 2, 3.0, 3), (9, 12, 2, 2, 0.05, 0), (16, 33, 3, 3, 0.05, 3), (17, 12, 2, 2, 0.05, 0)])
def test_stage_by_tracer_count(ntr, nlev, order, nrk, w_amp, terrain):
    g, st = case(nlev, ntr, w_amp, terrain)
    opts = abi.make_opts(1800.0, nrk_scal=nrk, scal_order=order)
    out, sct = run(g, st, opts)
    check(out, oracle_lib.scalar_transport(abi.FortranGrid(g), opts, st.tracers, sct, st, fp64=True))


# the 32-column tiles' groups: the counts around 32, the first and last of 40
# and of 48 tracers a block, two blocks of 32 and of 40, and a level split
@pytest.mark.parametrize("ntr,order,ks,w_amp,terrain", [
    (17, 2, 1, 0.05, 0), (24, 3, 1, 3.0, 3), (25, 2, 1, 0.05, 0), (33, 3, 1, 0.05, 3), (40, 2, 1, 3.0, 0),
    (41, 2, 1, 0.05, 3), (48, 3, 1, 0.05, 0), (49, 2, 1, 0.05, 0), (56, 3, 1, 0.05, 3), (57, 2, 1, 0.05, 0),
    (74, 2, 1, 0.05, 3), (33, 2, 2, 0.05, 0)])
def test_tile_groups(ntr, order, ks, w_amp, terrain):
    g, st = case(12, ntr, w_amp, terrain)
    opts = abi.make_opts(1800.0, scal_order=order)
    out, sct = run(g, st, opts, shape=(32, 32, ks, 0))
    check(out, oracle_lib.scalar_transport(abi.FortranGrid(g), opts, st.tracers, sct, st, fp64=True))


# limited and unlimited tracers in one quad (pdef), ragged counts, implicit
# columns, terrain
@pytest.mark.parametrize("monot,ntr,order,w_amp,terrain", [
    (2, 1, 2, 0.05, 0), (2, 6, 3, 3.0, 0), (2, 5, 2, 0.05, 3), (1, 3, 2, 3.0, 0), (1, 9, 3, 0.05, 3)])
def test_limited_stage(monot, ntr, order, w_amp, terrain):
    g, st = case(33, ntr, w_amp, terrain)
    pdef = [1 if n % 3 else 0 for n in range(ntr)] if monot == 2 and ntr > 1 else [1] * ntr
    opts = abi.make_opts(1800.0, scal_order=order, iscal_monot=monot)
    out, sct = run(g, st, opts, pdef=pdef)
    ref = [oracle_lib.scalar_transport(abi.FortranGrid(g), abi.make_opts(1800.0, scal_order=order,
                                                                         iscal_monot=monot if p or monot == 1 else 0),
                                       [t], [s], st, fp64=True)[0]
           for t, s, p in zip(st.tracers, sct, pdef)]
    check(out, ref)


# the per-call step in groups: the first count above a group, a ragged last
# group, and the last count before the wide groups
@pytest.mark.parametrize("ntr,order,w_amp", [(9, 2, 0.05), (21, 3, 3.0), (64, 2, 0.05)])
def test_per_call_groups(ntr, order, w_amp):
    g, st = case(12, ntr, w_amp, 0)
    opts = abi.make_opts(1800.0, scal_order=order)
    out, sct = run(g, st, opts, coherence=abi.SYNC_EACH_CALL)
    check(out, oracle_lib.scalar_transport(abi.FortranGrid(g), opts, st.tracers, sct, st, fp64=True))


# three calls in a row (the rotation buffers change roles) equal three
# resident steps; columns that are not prognosed -- the dummy point, and with
# a third of the others left out of jtw_prog those -- keep their values
@pytest.mark.parametrize("nrk", [2, 3])
@pytest.mark.parametrize("ntr,border", [(21, False), (21, True), (70, True)])
def test_per_call_groups_over_several_steps(ntr, border, nrk):
    g, st = case(12, ntr, 0.05, 0)
    opts = abi.make_opts(1800.0, nrk_scal=nrk)
    kept = np.arange(g.mwa) % 3 == 1 if border else np.arange(g.mwa) == 0
    out = []
    for coherence in (abi.SYNC_EACH_CALL, abi.RESIDENT):
        fg = abi.FortranGrid(g)
        table = np.ascontiguousarray(np.flatnonzero(~kept)[1 if border else 0:] + 1, dtype=np.int32)
        fg.struct.nw_prog, fg.struct.jtw_prog = table.size, abi.ptr(table, ctypes.c_int)
        dev = OlamGpu(fg, opts, HostState(vmasc=st.vmasc, wmasc=st.wmasc, rho=st.rho, wc=st.wc))
        try:
            dev.set_coherence(coherence)
            var_p = [t.copy() for t in st.tracers]
            dev.register_scalars(var_p, [np.zeros_like(t) for t in var_p])
            for _ in range(1 if border else 3):
                dev.scalar_transport_rk(st.rho_old)
            if coherence == abi.RESIDENT:
                dev.sync_to_host(abi.F_SCALARS)
            out.append(var_p)
        finally:
            dev.close()
    for n in range(ntr):
        if not border:
            assert relerr(out[0][n][1:], out[1][n][1:]) < 1e-6, n
        for o in out:
            assert np.array_equal(o[n][kept], st.tracers[n][kept]), n


# above 64 tracers on grids where the timed shapes are close, so that any of
# them may be chosen, 8-column tiles too (which have no group of 64 tracers);
# forced 8-column tiles take the step in one piece
@pytest.mark.parametrize("nlev", [5, 7, 10, 14])
@pytest.mark.parametrize("shape", [None, (8, 128, 1, 0)])
def test_per_call_wide_groups(nlev, shape):
    g, st = case(nlev, 70, 0.05, 0)
    opts = abi.make_opts(1800.0)
    out, sct = run(g, st, opts, coherence=abi.SYNC_EACH_CALL, shape=shape)
    check(out, oracle_lib.scalar_transport(abi.FortranGrid(g), opts, st.tracers, sct, st, fp64=True))


# mza = nlev + 1 at the sizes where the rows per lane and the warps per column
# change, with and without the column kernel's folded set-up
@pytest.mark.parametrize("nlev,kw", [(31, {}), (32, {}), (63, {}), (64, {}), (32, dict(ithil_monot=1))])
def test_acoustic_step_by_level_count(nlev, kw):
    g, ds = dyn_case(nxp=4, nlev=nlev, seed=8)
    fg = abi.FortranGrid(g)
    assert g.mza == nlev + 1
    opts = abi.make_opts(300.0, nacoust=4, **kw)
    arrays = oracle_lib.dyn_arrays(g, ds)
    o64, _ = oracle_long_steps(fg, opts, arrays, 1, True)
    o32, _ = oracle_long_steps(fg, opts, arrays, 1, False)
    hs, _ = gpu_long_steps(fg, opts, arrays, 1, abi.SYNC_EACH_CALL)
    check_fields(hs, o32, o64)


# the tables' entries past a column's npoly are the caller's padding: NaN
# there reaches no result
@pytest.mark.parametrize("order", [2, 3])
def test_padding_of_the_edge_tables_is_not_used(order):
    import copy
    from test_timestep_gpu import Dev, _case, _same
    g0, _, arrays, tr = _case(ntr=3)
    past = np.arange(7)[None, :] >= g0.npoly[:, None]
    g1 = copy.copy(g0)
    for k in ("gxps_coef", "gyps_coef", "xy_h", "xy_hu", "dirv", "xx_yy", "ecvec_vx", "ecvec_vy", "ecvec_vz"):
        a = getattr(g0, k).copy()
        a[past] = np.nan
        setattr(g1, k, a)
    opts = abi.make_opts(600.0, nacoust=2, scal_order=order, thil_order=order, wind_order=order)
    out = []
    for g in (g0, g1):
        d = Dev(g, arrays, tr, opts)
        try:
            d.dev.timestep(0)
            out.append(d.host())
        finally:
            d.close()
    assert all(np.isfinite(out[0][k]).all() for k in out[0])
    _same(out[0], out[1])


# M-point floors of their own on a grid whose W and V floors are all level 2:
# the level-3 vorticity damping takes its second-order plane below them
def test_m_floors_on_a_flat_grid():
    import copy
    g0, ds = dyn_case()
    g = copy.copy(g0)
    g.lpm = g0.lpm.copy()
    g.lpm[1::3] = 6
    opts = abi.make_opts(600.0, nacoust=4)
    assert opts.vort_damp_level == 3 and (g.lpw[1:] == 2).all() and (g.lpv[1:] == 2).all()
    fg = abi.FortranGrid(g)
    arrays = oracle_lib.dyn_arrays(g, ds)
    o64, _ = oracle_long_steps(fg, opts, arrays, 1, True)
    o32, _ = oracle_long_steps(fg, opts, arrays, 1, False)
    hs, _ = gpu_long_steps(fg, opts, arrays, 1, abi.SYNC_EACH_CALL)
    check_fields(hs, o32, o64)
