"""GPU test of olamgpu_update_scalar_noalloc, the stage entry point that
allocates nothing: two stages through it in a row reproduce one RK2
scalar_transport_rk of the library's plain form, and the two calls leave the
device's free memory unchanged.  Collected last so it also runs after every
other GPU test in the same process."""
import ctypes as C

import numpy as np
import pytest

from conftest import relerr, small_case
from olam_b200 import abi
from olam_b200.lib import HostState, OlamGpu, check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,terrain", [(2, 0), (3, 0), (2, 3)])
def test_noalloc_two_stages_match_transport(order, terrain):
    import torch
    g, st = small_case(nxp=6, nlev=12, ntr=1, seed=31)
    if terrain:
        from olam_b200.synth.grid import with_terrain
        g = with_terrain(g, terrain)                   # lpw / lpv floors of a mountain
    opts = abi.make_opts(1800.0, scal_order=order)    # RK2, no limiter
    fg = abi.FortranGrid(g)
    hs = HostState(vmasc=st.vmasc, wmasc=st.wmasc, rho=st.rho, wc=st.wc)
    dev = OlamGpu(fg, opts, hs)
    try:
        dev.set_transport_form(abi.TRANSPORT_PLAIN)
        var_p = [np.ascontiguousarray(st.tracers[0].copy())]
        var_t = [np.ascontiguousarray(st.sct[0].copy())]
        dev.register_scalars(var_p, var_t)
        diag = dev.scalar_transport_rk(st.rho_old, want_diag=True)
        assert diag.cfl_max < 0.9, "case must keep every column explicit"
        ref = var_p[0].copy()

        # device arrays owned by the caller (allocated here, not by the call)
        def dv(a):
            return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()
        scp0, sct = dv(st.tracers[0]), dv(st.sct[0])
        rhos = dv(st.rho.astype(np.float32))           # rhos(:,:,nrk) of RK2 = real(rho)
        vm, wm = dv(st.vmasc), dv(st.wmasc)
        s1, s2 = torch.zeros_like(scp0), torch.zeros_like(scp0)
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        L = dev.lib
        p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
        dtl = np.float32(opts.dtlm)

        def stage(src, dtr, dst):
            check(L.olamgpu_update_scalar_noalloc(p(src), p(scp0), p(sct), p(rhos), p(vm), p(wm),
                                                  C.c_float(dtr), p(dst), stream))

        stage(scp0, dtl * np.float32(0.5), s1)         # first call on the device: set-up
        torch.cuda.synchronize()
        free0 = torch.cuda.mem_get_info()[0]
        for _ in range(2):                             # two full passes, each two calls in a row
            stage(scp0, dtl * np.float32(0.5), s1)
            stage(s1, dtl * np.float32(1.0), s2)
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] == free0
        out = s2.cpu().numpy()
    finally:
        dev.close()
    e = relerr(out[1:], ref[1:])
    assert e < 1e-6, e


def test_noalloc_rejects_null_arrays():
    g, st = small_case(nxp=4, nlev=8, ntr=1)
    fg = abi.FortranGrid(g)
    dev = OlamGpu(fg, abi.make_opts(1800.0), HostState(vmasc=st.vmasc, wmasc=st.wmasc, rho=st.rho))
    try:
        rc = dev.lib.olamgpu_update_scalar_noalloc(None, None, None, None, None, None, C.c_float(1.0),
                                                   None, None)
        assert rc == abi.E_ARG
    finally:
        dev.close()


def test_noalloc_rejects_a_grid_beyond_the_scratch():
    # NXP = 75 with 60 levels at order 2 needs 50 NXP^2 mza + ... > 16 Mi floats
    from olam_b200.synth.grid import build_grid, stretched_levels
    from olam_b200.synth.state import transport_state
    g = build_grid(75, stretched_levels(60, 100.0, 30000.0), seed=5)
    st = transport_state(g, 600.0, 0, seed=5)
    fg = abi.FortranGrid(g)
    dev = OlamGpu(fg, abi.make_opts(600.0), HostState(vmasc=st.vmasc, wmasc=st.wmasc, rho=st.rho))
    try:
        import torch
        a = torch.zeros(g.mwa * g.mza, dtype=torch.float32, device="cuda")
        v = torch.zeros(g.mva * g.mza, dtype=torch.float32, device="cuda")
        p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
        rc = dev.lib.olamgpu_update_scalar_noalloc(p(a), p(a), p(a), p(a), p(v), p(a), C.c_float(1.0),
                                                   p(a), None)
        assert rc == abi.E_ARG
        assert b"scratch" in dev.lib.olamgpu_strerror(rc)
    finally:
        dev.close()


@pytest.mark.parametrize("order,terrain,alias", [(2, 0, "scp"), (3, 3, "scp"), (2, 3, "both"), (2, 0, "scp0")])
def test_noalloc_in_place(order, terrain, alias):
    """The result over scp (and, with "both", over scp0 at once), or over
    scp0, equals the result in an array of its own; columns outside jtw_prog
    stay as they were."""
    import torch
    g, st = small_case(nxp=6, nlev=40, ntr=1, seed=31)
    if terrain:
        from olam_b200.synth.grid import with_terrain
        g = with_terrain(g, terrain)
    dev = OlamGpu(abi.FortranGrid(g), abi.make_opts(1800.0, scal_order=order),
                  HostState(vmasc=st.vmasc, wmasc=st.wmasc, rho=st.rho, wc=st.wc))
    try:
        def dv(a):
            return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()
        a, sct, rhos = dv(st.tracers[0]), dv(st.sct[0]), dv(st.rho)
        vm, wm = dv(st.vmasc), dv(st.wmasc)
        a[0] = 7.0
        b = a if alias == "both" else a * 1.001

        def stage(scp, scp0, out):
            p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
            check(dev.lib.olamgpu_update_scalar_noalloc(p(scp), p(scp0), p(sct), p(rhos), p(vm), p(wm),
                                                        C.c_float(900.0), p(out),
                                                        C.c_void_p(torch.cuda.current_stream().cuda_stream)))

        ref = torch.zeros_like(a)
        stage(a, b, ref)
        for _ in range(3):
            s = a.clone()
            s0 = s if alias == "both" else b.clone()
            out = s0 if alias == "scp0" else s
            kept = out[0].clone()
            stage(s, s0, out)
            assert torch.equal(out[1:], ref[1:])
            assert torch.equal(out[0], kept)
    finally:
        dev.close()


@pytest.mark.parametrize("order", [2, 3])
def test_grid_without_the_jtw_wadj_table(order):
    """On a domain without borders jtw_wadj names no column that jtw_prog
    does not: a grid without it takes the no-allocation stage and the
    resident step with few tracers, with the results it has with the table."""
    import torch
    g, st = small_case(nxp=6, nlev=12, ntr=4, seed=31)
    out = []
    for table in (True, False):
        fg = abi.FortranGrid(g)
        if not table:
            fg.struct.nw_wadj, fg.struct.jtw_wadj = 0, None
        dev = OlamGpu(fg, abi.make_opts(1800.0, scal_order=order),
                      HostState(vmasc=st.vmasc, wmasc=st.wmasc, rho=st.rho, wc=st.wc))
        try:
            def dv(a):
                return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()
            arrays = [dv(a) for a in (st.tracers[0], st.tracers[0], st.sct[0], st.rho, st.vmasc, st.wmasc)]
            res = torch.zeros_like(arrays[0])
            p = [C.c_void_p(a.data_ptr()) for a in arrays + [res]]
            check(dev.lib.olamgpu_update_scalar_noalloc(*p[:6], C.c_float(900.0), p[6],
                                                        C.c_void_p(torch.cuda.current_stream().cuda_stream)))
            dev.set_coherence(abi.RESIDENT)
            var_p = [t.copy() for t in st.tracers]
            dev.register_scalars(var_p, [t.copy() for t in st.sct])
            dev.scalar_transport_rk(st.rho_old)
            dev.sync_to_host(abi.F_SCALARS)
            out.append((res.cpu().numpy(), var_p))
        finally:
            dev.close()
    assert np.array_equal(out[0][0], out[1][0])
    for a, b in zip(out[0][1], out[1][1]):
        assert relerr(b[1:], a[1:]) < 1e-6


@pytest.mark.parametrize("order,terrain", [(2, 0), (3, 3)])
def test_noalloc_nan_and_infinity_reach_their_stencil_only(order, terrain):
    """One stage of a tracer with NaN and infinite cells: the cells that are
    not finite after it are those whose stencil (upwind reconstruction at the
    six faces and the two W faces) holds one, found in numpy; all others have
    the value that a finite tracer gives."""
    import torch
    g, st = small_case(nxp=6, nlev=14, ntr=1, seed=31)
    if terrain:
        from olam_b200.synth.grid import with_terrain
        g = with_terrain(g, terrain)
    rng = np.random.default_rng(2)
    scp = st.tracers[0].copy()
    bad = np.zeros(scp.shape, bool)
    iw = rng.choice(np.arange(1, g.mwa), 12, replace=False)
    kb = g.lpw[iw] - 1
    k = rng.integers(kb, g.mza)
    bad[iw, k] = True
    dev = OlamGpu(abi.FortranGrid(g), abi.make_opts(1800.0, scal_order=order),
                  HostState(vmasc=st.vmasc, wmasc=st.wmasc, rho=st.rho, wc=st.wc))
    try:
        def stage(q):
            def dv(a):
                return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()
            arrays = [dv(a) for a in (q, st.tracers[0], st.sct[0], st.rho, st.vmasc, st.wmasc)]
            arrays.append(torch.zeros_like(arrays[0]))
            check(dev.lib.olamgpu_update_scalar_noalloc(*[C.c_void_p(a.data_ptr()) for a in arrays[:6]],
                                                        C.c_float(900.0), C.c_void_p(arrays[6].data_ptr()),
                                                        C.c_void_p(torch.cuda.current_stream().cuda_stream)))
            return arrays[6].cpu().numpy()
        ref = stage(scp)
        scp[iw, k] = np.where(np.arange(12) % 3 == 0, np.inf, np.nan)
        out = stage(scp)
    finally:
        dev.close()
    # the cells whose value a cell's gradient or its own value takes
    grad = bad.copy()
    for n in range(7):
        use = (n < g.npoly)[:, None] & (np.arange(g.mza)[None, :] >= g.lpv[g.itab_w_iv[:, n]][:, None] - 1)
        grad |= use & bad[g.itab_w_iw[:, n]]
    hit = np.zeros_like(bad)
    for w in range(1, g.mwa):
        b0 = g.lpw[w] - 1
        for lev in range(b0, g.mza):
            for n in range(g.npoly[w]):
                v = g.itab_w_iv[w, n]
                if lev >= g.lpv[v] - 1:
                    hit[w, lev] |= grad[g.itab_v_iw[v, 1 if st.vmasc[v, lev] < 0 else 0], lev]
            for f in (lev - 1, lev):                    # the W faces below and above
                if f < b0 or f == g.mza - 1:
                    hit[w, lev] |= bad[w, lev]
                    continue
                c = f + 1 if st.wmasc[w, f] < 0 else f
                hit[w, lev] |= bad[w, max(c - 1, b0):min(c + 2, g.mza)].any()
    for w in range(1, g.mwa):
        hit[w, :g.lpw[w] - 1] = hit[w, g.lpw[w] - 1]
    assert np.array_equal(~np.isfinite(out[1:]), hit[1:])
    assert np.array_equal(out[1:][~hit[1:]], ref[1:][~hit[1:]])


def test_noalloc_recorded_by_the_caller():
    """Two stages and a caller's own operation between them recorded into a
    CUDA graph, the second stage in place; the replay on new inputs equals
    the calls made one by one."""
    import torch
    g, st = small_case(nxp=6, nlev=40, ntr=2, seed=31)
    dev = OlamGpu(abi.FortranGrid(g), abi.make_opts(1800.0),
                  HostState(vmasc=st.vmasc, wmasc=st.wmasc, rho=st.rho, wc=st.wc))
    try:
        def dv(a):
            return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()
        scp, sct, rhos, vm, wm = dv(st.tracers[0]), dv(st.sct[0]), dv(st.rho), dv(st.vmasc), dv(st.wmasc)
        mid = torch.zeros_like(scp)

        def stage(src, dst):
            p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
            check(dev.lib.olamgpu_update_scalar_noalloc(p(src), p(scp), p(sct), p(rhos), p(vm), p(wm), C.c_float(900.0),
                                                        p(dst), C.c_void_p(torch.cuda.current_stream().cuda_stream)))

        def both():
            stage(scp, mid)
            mid.mul_(1.001)
            stage(mid, mid)

        both()                                         # first call: set-up
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            both()
        for n in (1, 0):
            scp.copy_(dv(st.tracers[n]))
            both()
            ref = mid.clone()
            mid.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(mid[1:], ref[1:])
    finally:
        dev.close()
