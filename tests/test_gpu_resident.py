"""The solvers that keep their search direction in shared memory, bit for bit
against the oracle at the sizes where their forms change: one tree block up to
12 (a cluster; 2,048 nodes per block), 13 to 24 (tagged partial sums), more
(an arrival counter), more tree blocks than SMs (two per physical block), with
uneven last blocks, unstructured node degrees (odd slice widths) and both
storages.  Iterations are capped: every form runs a few dozen."""
import ctypes

import numpy as np
import pytest

from opentelemac_b200 import _native, bief, meshgen as mg

pytestmark = pytest.mark.gpu


def _grid(nx, ny, seed=3):
    """nx x ny jittered grid, quads cut along random diagonals."""
    rng = np.random.default_rng([seed, nx, ny])
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="xy")
    x = ((i + rng.uniform(-0.2, 0.2, i.shape)) / nx).ravel()
    y = ((j + rng.uniform(-0.2, 0.2, i.shape)) / nx).ravel()
    a = (np.arange(ny - 1)[:, None] * nx + np.arange(nx - 1)).ravel()
    b, c, d = a + 1, a + nx + 1, a + nx
    cut = (rng.random(a.size) < 0.5)[:, None]
    ik = np.empty((2 * a.size, 3), dtype=np.int32)
    ik[0::2] = np.where(cut, np.stack([a, b, d], 1), np.stack([a, b, c], 1))
    ik[1::2] = np.where(cut, np.stack([b, c, d], 1), np.stack([a, c, d], 1))
    return x, y, ik


# (nx, ny, tree blocks)
SIZES = [(2, 2, 1), (5, 7, 1), (32, 64, 1), (33, 63, 2), (128, 128, 8), (129, 128, 9),
         (192, 128, 12), (193, 128, 13), (224, 219, 24), (225, 221, 25)]


def _problem(oracle_mod, x, y, ik, seed=1):
    dm, xm = oracle_mod.wave_matrix(x, y, ik, mg.wave_coef(mg.depth_smooth(x, y, ik)))
    xt = np.random.default_rng(seed).uniform(-1, 1, x.size)
    b = oracle_mod.matvec("X=AY    ", ik, dm, "Q", xm, "S", xt)
    return dm, xm, b


def _stored(oracle_mod, ik, n, dm, xm, typext, storage, bps=0):
    mesh = bief.Mesh(ik, n)
    if bps:
        mesh.set_blocks_per_sm(bps)
    A = bief.Matrix(mesh, dm, xm, "Q", typext)
    seg = None
    if storage == "seg":
        g1, g2, es, ori = mg.segments(ik, n)
        mesh.set_segments(g1, g2)
        A.to_segments()
        seg = (g1, g2, oracle_mod.assex3(es, ori, typext, xm, g1.size))
    return mesh, A, seg


def _check_solve(oracle_mod, ik, n, dm, xm, typext, b, storage, slv, nitmax, x0, modass=1, bps=0):
    mesh, A, seg = _stored(oracle_mod, ik, n, dm, xm, typext, storage, bps)
    G, T = mesh.launch_info()
    x = x0.copy()
    cfg = bief.SlvCfg(slv=slv, nitmax=nitmax, precon=2, krylov=0, eps=1e-9, zero=0.0)
    st, nit, relres = bief.solve(x, A, b.copy(), cfg, modass=modass)
    mode = oracle_mod.DOT_BLOCKED if modass == 1 else oracle_mod.DOT_COMP_BLOCKED
    kw = dict(slv=slv, eps=1e-9, nitmax=nitmax, x0=x0, dot_mode=mode, nblocks=G, nthreads=T)
    with oracle_mod.threads():
        if seg:
            r = oracle_mod.solve_seg(seg[0], seg[1], dm, "Q", seg[2], typext, b, **kw)
        else:
            r = oracle_mod.solve(ik, dm, "Q", xm, typext, b, **kw)
    assert (st, nit, relres) == (r["status"], r["nit"], r["relres"])
    np.testing.assert_array_equal(x, r["x"])
    # again on the same handle, the plan in place
    x = x0.copy()
    assert bief.solve(x, A, b.copy(), cfg, modass=modass)[1] == nit
    np.testing.assert_array_equal(x, r["x"])
    mesh.close()
    return G


def _check_mixed(oracle_mod, ik, n, dm, xm, b, storage, max_inner, bps=0):
    mesh, A, seg = _stored(oracle_mod, ik, n, dm, xm, "S", storage, bps)
    G, T = mesh.launch_info()
    x = np.zeros(n)
    st, outer, inner, relres = bief.solve_mixed(x, A, b, precon=2, inner_tol=0.1,
                                                outer_tol=1e-10, max_inner=max_inner)
    kw = dict(precon=2, inner_tol=0.1, outer_tol=1e-10, max_outer=1000, max_inner=max_inner,
              nblocks=G, nthreads=T)
    with oracle_mod.threads():
        if seg:
            r = oracle_mod.solve_mixed_seg(seg[0], seg[1], dm, "Q", seg[2], b, **kw)
        else:
            r = oracle_mod.solve_mixed(ik, dm, "Q", xm, b, **kw)
    assert (st, outer, inner, relres) == (r["status"], r["outer"], r["inner"], r["relres"])
    np.testing.assert_array_equal(x, r["x"])
    # the binary32 product rebuilds its own slots after the solve's paired ones
    import torch
    xs = torch.tensor(b, device="cuda", dtype=torch.float32)
    y1, y2 = torch.empty_like(xs), torch.empty_like(xs)
    bief.matvec32(y1, A, xs)
    bief.solve_mixed(np.zeros(n), A, b, precon=2, inner_tol=0.1, outer_tol=1e-10, max_inner=3)
    bief.matvec32(y2, A, xs)
    assert torch.equal(y1, y2)
    mesh.close()


@pytest.mark.parametrize("storage", ["ebe", "seg"])
@pytest.mark.parametrize("nx,ny,blocks", SIZES)
def test_forms_bitexact(oracle_mod, nx, ny, blocks, storage):
    x, y, ik = _grid(nx, ny)
    n = x.size
    dm, xm, b = _problem(oracle_mod, x, y, ik)
    x0 = np.random.default_rng(5).uniform(-0.1, 0.1, n)
    assert _check_solve(oracle_mod, ik, n, dm, xm, "S", b, storage, 1, 40, x0) == blocks
    _check_mixed(oracle_mod, ik, n, dm, xm, b, storage, 60)


@pytest.mark.parametrize("modass", [1, 3])
@pytest.mark.parametrize("typext,storage", [("S", "ebe"), ("Q", "ebe"), ("Q", "seg")])
def test_cgstab_bitexact(oracle_mod, typext, storage, modass):
    """CGSTAB's shared-memory form (13 tree blocks and more)."""
    x, y, ik = _grid(171, 161)
    n = x.size
    dm, xm, b = _problem(oracle_mod, x, y, ik)
    if typext == "Q":
        rng = np.random.default_rng(2)
        xm = np.concatenate([xm, xm * (1 + 0.05 * rng.uniform(-1, 1, xm.shape))])
    assert _check_solve(oracle_mod, ik, n, dm, xm, typext, b, storage, 6, 25, np.zeros(n),
                        modass) > 12


@pytest.mark.parametrize("npts", [3000, 28000, 60000])
def test_random_numbering(oracle_mod, npts):
    """Points numbered at random: the halo is most of the mesh."""
    x, y, ik = mg.delaunay_mesh(npts)
    n = x.size
    dm, xm, b = _problem(oracle_mod, x, y, ik)
    _check_solve(oracle_mod, ik, n, dm, xm, "S", b, "ebe", 1, 25, np.zeros(n))
    _check_mixed(oracle_mod, ik, n, dm, xm, b, "ebe", 30)


def test_two_tree_blocks_per_block(oracle_mod):
    """More tree blocks than SMs (two blocks per SM asked for on a mesh of an
    odd number of them): two tree blocks per physical block, the last alone."""
    x, y, ik = _grid(601, 599)
    n = x.size
    dm, xm, b = _problem(oracle_mod, x, y, ik)
    G = _check_solve(oracle_mod, ik, n, dm, xm, "S", b, "ebe", 1, 8, np.zeros(n), bps=2)
    assert G > 148
    _check_mixed(oracle_mod, ik, n, dm, xm, b, "ebe", 12, bps=2)


def test_zero_rhs_and_breakdown(oracle_mod):
    """B = 0 and an indefinite matrix, in each form."""
    for nx, ny in ((20, 21), (171, 161), (240, 230)):
        x, y, ik = _grid(nx, ny)
        n = x.size
        dm, xm, b = _problem(oracle_mod, x, y, ik)
        mesh = bief.Mesh(ik, n)
        A = bief.Matrix(mesh, dm, xm, "Q", "S")
        cfg = bief.SlvCfg(slv=1, nitmax=50, precon=2, krylov=0, eps=1e-8, zero=0.0)
        u = np.ones(n)
        assert bief.solve(u, A, np.zeros(n), cfg)[:2] == (0, 0) and not u.any()
        u = np.ones(n)
        assert bief.solve_mixed(u, A, np.zeros(n))[0] == 0 and not u.any()
        A.set(dm, 3.0 * xm, "Q", "S")
        with pytest.raises(bief.BiefError):
            bief.solve(np.zeros(n), A, b.copy(), cfg)
        mesh.close()


@pytest.mark.parametrize("nx,ny", [(60, 61), (171, 161), (251, 241)])
def test_segments_that_are_no_face(oracle_mod, nx, ny):
    """A segment need not be an element's face: its far node belongs to the
    halo all the same (each form; GRACJG, CGSTAB and the mixed solve)."""
    x, y, ik = _grid(nx, ny)
    n = x.size
    dm, xm, _ = _problem(oracle_mod, x, y, ik)
    g1, g2, es, ori = mg.segments(ik, n)
    xa = oracle_mod.assex3(es, ori, "S", xm, g1.size)
    face = set(zip(np.minimum(g1, g2).tolist(), np.maximum(g1, g2).tolist()))
    rng = np.random.default_rng(nx)
    far = [(0, n - 1), (n // 2, 1), (n - 2, n // 3)]  # and at random over the mesh
    for a, b in rng.integers(0, n, (40, 2)).tolist():
        k = (min(a, b), max(a, b))
        if a != b and k not in face and k not in {(min(p), max(p)) for p in far}:
            far.append((a, b))
    g1 = np.concatenate([g1, [p[0] for p in far]])
    g2 = np.concatenate([g2, [p[1] for p in far]])
    xa = np.concatenate([xa.ravel(), -0.3 * dm.mean() * rng.uniform(0.5, 1.0, len(far))])
    dm = dm.copy()
    for a, b in far:  # diagonally as dominant as before
        dm[a] += 0.4 * dm.mean()
        dm[b] += 0.4 * dm.mean()
    b = rng.uniform(-1, 1, n) * dm
    mesh = bief.Mesh(ik, n)
    mesh.set_segments(g1, g2)
    A = bief.Matrix(mesh).set_seg(dm, xa)
    G, T = mesh.launch_info()
    for slv in (1, 6):
        u = np.zeros(n)
        cfg = bief.SlvCfg(slv=slv, nitmax=25, precon=2, krylov=0, eps=1e-9, zero=0.0)
        st, nit, relres = bief.solve(u, A, b.copy(), cfg)
        with oracle_mod.threads():
            r = oracle_mod.solve_seg(g1, g2, dm, "Q", xa, "S", b, slv=slv, eps=1e-9, nitmax=25,
                                     dot_mode=oracle_mod.DOT_BLOCKED, nblocks=G, nthreads=T)
        assert (st, nit, relres) == (r["status"], r["nit"], r["relres"])
        np.testing.assert_array_equal(u, r["x"])
    u = np.zeros(n)
    got = bief.solve_mixed(u, A, b, inner_tol=0.1, outer_tol=1e-10, max_inner=40)
    with oracle_mod.threads():
        r = oracle_mod.solve_mixed_seg(g1, g2, dm, "Q", xa, b, inner_tol=0.1, outer_tol=1e-10,
                                       max_inner=40, nblocks=G, nthreads=T)
    assert got == (r["status"], r["outer"], r["inner"], r["relres"])
    np.testing.assert_array_equal(u, r["x"])
    mesh.close()


def test_threads_with_their_own_handles():
    """Two host threads, each with a mesh and a stream of its own: the launch
    of one must not depend on the shared memory that the other's mesh asks
    for (both meshes run the same kernel)."""
    import threading
    import torch
    todo = []
    for nx in (41, 90):
        x, y, ik = _grid(nx, nx)
        n = x.size
        mesh = bief.Mesh(ik, n)
        A = bief.Matrix(mesh, np.full(n, 8.0), np.full((3, ik.shape[0]), -0.5), "Q", "S")
        b = torch.rand(n, device="cuda", dtype=torch.float64)
        u = torch.empty_like(b)
        todo.append((mesh, A, b, u, torch.cuda.Stream()))
    torch.cuda.synchronize()
    errors = []
    start = threading.Barrier(len(todo))

    def work(mesh, A, b, u, stream):
        cfg = bief.SlvCfg(slv=1, nitmax=2, precon=2, krylov=0, eps=1e-12, zero=0.0)
        try:
            with torch.cuda.stream(stream):
                start.wait()
                ref = None
                for _ in range(1000):
                    u.zero_()
                    bief.solve(u, A, b, cfg)
                    if ref is None:
                        ref = u.clone()
                assert torch.equal(u, ref)
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=a) for a in todo]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    # whichever solved last, the kernel's limit is the device's
    limit = ctypes.c_int()
    bief.solve(todo[0][3], todo[0][1], todo[0][2],
               bief.SlvCfg(slv=1, nitmax=2, precon=2, krylov=0, eps=1e-12, zero=0.0))
    assert _native.lib().bief_selftest_smem(0, ctypes.byref(limit)) == 0
    assert limit.value == torch.cuda.get_device_properties(0).shared_memory_per_block_optin
    for a in todo:
        a[0].close()


def test_no_memory_for_the_plan():
    """A device with no memory left for a solver's plan: the kernels that need
    none solve instead, with the same bits."""
    import torch
    nx, ny = 2001, 1001
    k = np.arange(nx * ny).reshape(ny, nx)
    a, b, c, d = (v.ravel() for v in (k[:-1, :-1], k[:-1, 1:], k[1:, 1:], k[1:, :-1]))
    ik = np.concatenate([np.stack([a, b, c], 1), np.stack([a, c, d], 1)]).astype(np.int32)
    n = nx * ny
    rhs = torch.rand(n, device="cuda", dtype=torch.float64)

    def handle():
        mesh = bief.Mesh(ik, n)
        return bief.Matrix(mesh, np.full(n, 8.0), np.full((3, ik.shape[0]), -0.5), "Q", "S")

    def cg(A, u):
        cfg = bief.SlvCfg(slv=1, nitmax=10, precon=2, krylov=0, eps=1e-13, zero=0.0)
        return bief.solve(u, A, rhs, cfg)

    def mixed(A, u):
        return bief.solve_mixed(u, A, rhs, max_inner=10)

    todo = [(f, handle(), torch.zeros_like(rhs)) for f in (cg, mixed)]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    fill = torch.empty(free - (24 << 20), device="cuda", dtype=torch.uint8)
    got = [f(A, u) for f, A, u in todo]
    del fill
    torch.cuda.empty_cache()
    A = handle()
    for (f, B, u), st in zip(todo, got):
        v = torch.zeros_like(rhs)
        assert f(A, v) == st
        assert torch.equal(u, v)
        B.mesh.close()
    A.mesh.close()


def _rows_mesh(nx, ny):
    k = np.arange(nx * ny).reshape(ny, nx)
    a, b, c, d = (v.ravel() for v in (k[:-1, :-1], k[:-1, 1:], k[1:, 1:], k[1:, :-1]))
    ik = np.concatenate([np.stack([a, b, c], 1), np.stack([a, c, d], 1)]).astype(np.int32)
    n = nx * ny
    mesh = bief.Mesh(ik, n)
    return bief.Matrix(mesh, np.full(n, 8.0), np.full((3, ik.shape[0]), -0.5), "Q", "S"), n


@pytest.mark.parametrize("nx,ny,slv,bps", [(70, 71, 6, 0), (601, 599, 6, 2), (2001, 2001, 1, 0)])
def test_no_plan_for_a_method_without_the_form(nx, ny, slv, bps):
    """CGSTAB on a cluster-sized mesh and with two tree blocks per block, and
    GRACJG on a mesh whose window cannot fit, solve without a plan: the first
    call launches what later ones do, and holds no memory for it."""
    import torch
    A, n = _rows_mesh(nx, ny)
    if bps:
        A.mesh.set_blocks_per_sm(bps)
    b = torch.rand(n, device="cuda", dtype=torch.float64)
    u = torch.zeros_like(b)
    cfg = bief.SlvCfg(slv=slv, nitmax=3, precon=2, krylov=0, eps=1e-13, zero=0.0)
    if slv == 6:  # its vectors are allocated at the first call
        bief.solve(u, A, b, bief.SlvCfg(slv=7, nitmax=1, precon=2, krylov=2, eps=1e-13, zero=0.0))
    torch.cuda.synchronize()
    free, launches = torch.cuda.mem_get_info()[0], []
    for _ in range(2):
        before = A.mesh.kernel_launches()
        bief.solve(u.zero_(), A, b, cfg)
        launches.append(A.mesh.kernel_launches() - before)
    assert launches[0] == launches[1]
    assert torch.cuda.mem_get_info()[0] == free
    A.mesh.close()


def test_plan_holds_one_list_per_kind_of_solve(oracle_mod):
    """Lists are made as solves ask for them, in any order of the kinds: the
    halo counted once (with the first), one launch for each list."""
    x, y, ik = _grid(171, 161)
    n = x.size
    dm, xm, b = _problem(oracle_mod, x, y, ik)
    g1, g2, es, ori = mg.segments(ik, n)
    cfg = bief.SlvCfg(slv=1, nitmax=20, precon=2, krylov=0, eps=1e-9, zero=0.0)

    def run(A, kind):
        u = np.zeros(n)
        before = A.mesh.kernel_launches()
        if kind == "cg":
            bief.solve(u, A, b.copy(), cfg)
        else:
            bief.solve_mixed(u, A, b, outer_tol=1e-10, max_inner=20)
        return u, A.mesh.kernel_launches() - before

    want = {}
    for order in (("cg", "mixed"), ("mixed", "cg")):
        mesh = bief.Mesh(ik, n)
        mesh.set_segments(g1, g2)
        A = bief.Matrix(mesh, dm, xm, "Q", "S")
        extra = []
        for storage in ("ebe", "seg"):
            if storage == "seg":
                A.to_segments()
            for kind in order:
                u, first = run(A, kind)
                v, later = run(A, kind)
                extra.append(first - later)
                np.testing.assert_array_equal(u, v)
                np.testing.assert_array_equal(u, want.setdefault((storage, kind), u))
        assert extra == [2, 1, 1, 1]
        mesh.close()


def _shuffled(x, y, ik, seed=7):
    """Nodes and elements in random order."""
    rng = np.random.default_rng(seed)
    new_id = rng.permutation(x.size)
    xs, ys = np.empty_like(x), np.empty_like(y)
    xs[new_id], ys[new_id] = x, y
    return xs, ys, new_id[ik[rng.permutation(ik.shape[0])]].astype(np.int32)


# GRACJG's and the mixed solve's form, iterations of each: more than two tree
# rows per thread in the last block (R = 3: no cluster); vectors in global
# memory; local indices as element numbers; two tree blocks per block
@pytest.mark.parametrize("nx,ny,shuffle,bps,storage,cg,mixed,its", [
    (63, 65, False, 0, "ebe", "tagged", "tagged", 40),
    (983, 25, False, 0, "seg", "tagged", "tagged", 40),
    (707, 709, True, 0, "ebe", "counter+global", "counter+elements", 10),
    (1301, 1307, False, 0, "ebe", "counter+global", "counter+global+elements", 10),
    (1301, 1307, False, 0, "seg", "counter+global", "counter+global+elements", 10),
    (601, 599, False, 2, "seg", "counter+two", "counter+two", 10),
    (1301, 1307, False, 2, "ebe", "counter+global+two", "counter+global+elements+two", 10)])
def test_large_forms_bitexact(oracle_mod, nx, ny, shuffle, bps, storage, cg, mixed, its):
    x, y, ik = _grid(nx, ny)
    if shuffle:
        x, y, ik = _shuffled(x, y, ik)
    n = x.size
    dm, xm, b = _problem(oracle_mod, x, y, ik)
    mesh, A, seg = _stored(oracle_mod, ik, n, dm, xm, "S", storage, bps)
    assert mesh.solve_form() is None
    G, T = mesh.launch_info()
    x0 = np.random.default_rng(5).uniform(-0.1, 0.1, n)
    cfg = bief.SlvCfg(slv=1, nitmax=its, precon=2, krylov=0, eps=1e-9, zero=0.0)
    kw = dict(eps=1e-9, nitmax=its, x0=x0, dot_mode=oracle_mod.DOT_BLOCKED, nblocks=G, nthreads=T)
    with oracle_mod.threads():
        r = (oracle_mod.solve_seg(seg[0], seg[1], dm, "Q", seg[2], "S", b, **kw) if seg else
             oracle_mod.solve(ik, dm, "Q", xm, "S", b, **kw))
    for _ in range(2):
        u = x0.copy()
        assert bief.solve(u, A, b.copy(), cfg) == (r["status"], r["nit"], r["relres"])
        np.testing.assert_array_equal(u, r["x"])
        assert mesh.solve_form() == cg
    kw = dict(precon=2, inner_tol=0.1, outer_tol=1e-10, max_outer=1000, max_inner=its, nblocks=G,
              nthreads=T)
    with oracle_mod.threads():
        r = (oracle_mod.solve_mixed_seg(seg[0], seg[1], dm, "Q", seg[2], b, **kw) if seg else
             oracle_mod.solve_mixed(ik, dm, "Q", xm, b, **kw))
    for _ in range(2):
        u = np.zeros(n)
        got = bief.solve_mixed(u, A, b, precon=2, inner_tol=0.1, outer_tol=1e-10, max_inner=its)
        assert got == (r["status"], r["outer"], r["inner"], r["relres"])
        np.testing.assert_array_equal(u, r["x"])
        assert mesh.solve_form() == mixed
    mesh.close()


@pytest.mark.parametrize("nx,ny,kind,form", [
    (40, 41, "cg", "cluster"), (171, 161, "cg", "tagged"), (225, 221, "cg", "counter"),
    (40, 41, "mixed", "cluster"), (171, 161, "mixed", "tagged"), (225, 221, "mixed", "counter"),
    (40, 41, "stab", "gather"), (171, 161, "stab", "counter"), (40, 41, "comp", "gather")])
def test_form_of_the_last_solve(nx, ny, kind, form):
    """The sizes of the tests above do run the forms that they are for."""
    A, n = _rows_mesh(nx, ny)
    u, b = np.zeros(n), np.ones(n)
    if kind == "mixed":
        bief.solve_mixed(u, A, b, max_inner=3)
    else:
        cfg = bief.SlvCfg(slv=6 if kind == "stab" else 1, nitmax=3, precon=2, krylov=0, eps=1e-9,
                          zero=0.0)
        bief.solve(u, A, b, cfg, modass=3 if kind == "comp" else 1)
    assert A.mesh.solve_form() == form
    A.mesh.close()
