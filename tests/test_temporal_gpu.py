"""Kernels that take several sweeps, or a whole iteration, per pass over memory,
at the edges of their tiles and rules: bit for bit against the oracle."""
import numpy as np
import pytest

import cfm
import oracle

pytestmark = pytest.mark.gpu


def rand_grid(shape, prec, seed):
    return np.random.default_rng(seed).uniform(-1, 1, shape).astype(cfm.np_dtype(prec))


# One tile, tile widths of 128 columns plus or minus one, several tiles of each kernel
# shape, a last tile of few columns, rows that are and are not a multiple of 16 bytes,
# and a grid beyond the chip (several strips and chunks of the streaming kernel).
@pytest.mark.parametrize("mirror", [False, True])
@pytest.mark.parametrize("prec", [cfm.FP64, cfm.FP32])
@pytest.mark.parametrize("shape,niter", [((18, 128), 9), ((66, 129), 18), ((67, 127), 33), ((260, 250), 26),
                                         ((515, 236), 17), ((300, 900), 25), ((2100, 2300), 12),
                                         ((1900, 2301), 11), ((9000, 70), 13), ((3, 4000), 10)])
def test_2d_several_sweeps_per_pass(shape, niter, prec, mirror):
    a = rand_grid(shape, prec, 31)
    with cfm.Jacobi(2, shape[1], shape[0], 1, prec, 1, cfm.JACOBI_PERSISTENT) as j:
        if mirror:
            j.set_boundary(cfm.BOUNDARY_MIRROR)
        j.upload(a)
        j.run(niter)
        want = (oracle.jacobi2d_mirror if mirror else oracle.jacobi2d)(a, niter)
        np.testing.assert_array_equal(j.download(), want)


# Runs of one and two sweeps among longer ones on one handle: on either side of the sizes from
# which short runs go to the row-marching kernel (that one sets the edge cells in a launch of its
# own), where the counters of the on-chip kernel go on from run to run.
@pytest.mark.parametrize("shape,prec,impl,marches", [
    ((700, 1000), cfm.FP64, cfm.JACOBI_PERSISTENT, (0, 0)), ((800, 1000), cfm.FP64, cfm.JACOBI_PERSISTENT, (0, 1)),
    ((800, 1000), cfm.FP64, cfm.JACOBI_RESIDENT, (0, 0)), ((800, 1001), cfm.FP64, cfm.JACOBI_PERSISTENT, (0, 0)),
    ((1300, 1160), cfm.FP32, cfm.JACOBI_PERSISTENT, (0, 1)), ((4900, 5000), cfm.FP64, cfm.JACOBI_PERSISTENT, (0, 0)),
    ((5100, 5000), cfm.FP64, cfm.JACOBI_PERSISTENT, (1, 1)), ((5100, 5000), cfm.FP64, cfm.JACOBI_RESIDENT, (1, 1))])
def test_2d_short_runs(shape, prec, impl, marches):
    a = rand_grid(shape, prec, 46)
    with cfm.Jacobi(2, shape[1], shape[0], 1, prec, 1, impl) as j:
        j.upload(a)
        counts = (2, 1, 9, 1, 2, 5, 2)
        for n in counts:
            assert j.run(n).launches == (1 + marches[n - 1] if n <= 2 else 1)
        np.testing.assert_array_equal(j.download(), oracle.jacobi2d(a, sum(counts)))


# Rows and columns at the tile edges (rows of a multiple of 16 bytes or not), z chunks that
# end beside the periodic planes, odd and even counts.
@pytest.mark.parametrize("py", [0, 1])
@pytest.mark.parametrize("prec", [cfm.FP64, cfm.FP32])
@pytest.mark.parametrize("shape,niter", [((9, 38, 64), 4), ((40, 39, 63), 5), ((12, 75, 65), 6),
                                         ((70, 40, 127), 3), ((33, 90, 129), 7), ((6, 5, 250), 8)])
def test_3d_two_sweeps_per_pass(shape, niter, prec, py):
    a = rand_grid(shape, prec, 32)
    nz, ny, nx = shape
    with cfm.Jacobi(3, nx, ny, nz, prec, py, cfm.JACOBI_PERSISTENT) as j:
        j.upload(a)
        j.run(niter)
        np.testing.assert_array_equal(j.download(), oracle.jacobi3d(a, niter, py))


# Short runs among longer ones on one handle, which take the one-sweep kernel by the sizes:
# passes of runs of 1, 2, 4 and 12 sweeps (the two-sweep kernel makes 1, 2, 3 and 7).
@pytest.mark.parametrize("shape,prec,passes", [
    ((40, 40, 40), cfm.FP64, (1, 2, 3, 7)), ((90, 100, 100), cfm.FP64, (1, 2, 3, 7)), ((250, 256, 256), cfm.FP64, (1, 2, 4, 7)),
    ((350, 256, 256), cfm.FP64, (1, 2, 3, 7)), ((250, 512, 256), cfm.FP32, (1, 2, 3, 7))])
def test_3d_short_runs(shape, prec, passes):
    a = rand_grid(shape, prec, 47)
    nz, ny, nx = shape
    with cfm.Jacobi(3, nx, ny, nz, prec, 1, cfm.JACOBI_PERSISTENT) as j:
        j.upload(a)
        points = np.prod([n - 2 for n in shape])
        for n, want in ((2, passes[1]), (1, passes[0]), (4, passes[2]), (12, passes[3]), (2, passes[1])):
            assert j.run(n).bytes == points * want * 2 * (8 if prec == cfm.FP64 else 4)
        np.testing.assert_array_equal(j.download(), oracle.jacobi3d(a, 21, 1))


def test_3d_launch_shape_is_that_of_the_sweep_order(monkeypatch):
    """Neighbourhood order runs on the one-sweep shape; rows that are not a multiple of 16
    bytes keep the two-sweep kernel."""
    def shape(nx):
        with cfm.Jacobi(3, nx, 40, 40, cfm.FP64, 1, cfm.JACOBI_PERSISTENT) as j:
            barrier = j.launch_shape(), cfm.lib.cfm_jacobi_zchunk(j.h)
            j.set_dataflow(True)
            return barrier, (j.launch_shape(), cfm.lib.cfm_jacobi_zchunk(j.h))
    two, order = shape(64)
    ragged = shape(63)
    monkeypatch.setenv("CFM_J3D_TMA_VARIANT", "0")
    one, _ = shape(64)
    assert order == one and order != two and ragged[0] == ragged[1]


def test_3d_two_sweeps_timeout_returns_status_and_handle_stays_usable(monkeypatch):
    """Waits far shorter than a plane's copy: the run ends with a status (every block lets
    its copies land first) and the handle's next run is right.  One column of 149 units,
    so on 148 SMs one block works twice as long as the others wait."""
    monkeypatch.setenv("CFM_J3D_ZCHUNK", "200")
    nx, ny, nz = 64, 30, 2 + 149 * 200
    with cfm.Jacobi(3, nx, ny, nz, cfm.FP64, 1, cfm.JACOBI_PERSISTENT) as j, \
            cfm.Jacobi(3, nx, ny, nz, cfm.FP64, 1, cfm.JACOBI_HOST_LOOP) as want:
        j.load_problem(cfm.PROBLEM_CONFIG)
        cfm.set_barrier_timeout_ms(1e-4)
        try:
            assert j.run(5, allowed=(cfm.BARRIER_TIMEOUT,)).status == cfm.BARRIER_TIMEOUT
        finally:
            cfm.set_barrier_timeout_ms(2000)
        for h in (j, want):
            h.load_problem(cfm.PROBLEM_CONFIG)
            h.run(5)
        np.testing.assert_array_equal(j.download(), want.download())


# One tile in all, one per block, two, three, four and six per block; systems whose rows all
# have neighbours in other blocks; beyond the chip.
@pytest.mark.parametrize("shape,maxiter", [((20, 30), 400), ((33, 31), 400), ((300, 200), 60), ((450, 500), 40),
                                           ((600, 640), 30), ((760, 700), 30), ((930, 900), 20), ((1100, 1000), 20),
                                           ((50, 50, 50), 60), ((80, 75, 70), 30), ((83, 83, 83), 20), ((100, 100, 90), 20)])
def test_cg_system_on_chip(shape, maxiter):
    k, f = cfm.varcoef_problem(shape, 33)
    dims = len(shape)
    grid = (shape[-1], shape[-2], shape[0] if dims == 3 else 1)
    xo, st_o, it_o, rs_o, _ = oracle.krylov_stencil(dims, grid, cfm.varcoef_coeffs(k), f, oracle.STD, maxiter, 1e-8)
    x, st = cfm.CG(cfm.Stencil(k), cfm.CG_PERSISTENT, maxiter, 1e-8).solve(f.ravel())
    assert st.status == st_o and st.iterations == it_o and st.refinements == rs_o
    np.testing.assert_array_equal(x, xo)


# Shapes whose dynamic shared memory on chip is exactly a block's 227 KB, which leaves no
# room for the kernel's static part: two in 2D (six tiles per block), two in 3D (four).
@pytest.mark.parametrize("shape", [(150, 4159), (215, 4159), (60, 176, 47), (56, 140, 59)])
def test_cg_on_chip_at_the_shared_memory_limit(shape):
    k, f = cfm.varcoef_problem(shape, 37)
    dims = len(shape)
    grid = (shape[-1], shape[-2], shape[0] if dims == 3 else 1)
    xo, _, it_o, _, _ = oracle.krylov_stencil(dims, grid, cfm.varcoef_coeffs(k), f, oracle.STD, 12, 0.0)
    x, st = cfm.CG(cfm.Stencil(k), cfm.CG_PERSISTENT, 12, 0.0).solve(f.ravel())
    assert st.iterations == it_o
    np.testing.assert_array_equal(x, xo)


# Handles of one kernel whose systems need different amounts of shared memory (narrower
# rows, or thinner planes, need less), the larger one solved after the smaller was created.
@pytest.mark.parametrize("large,small", [((480, 500), (1000, 240)), ((60, 60, 60), (240, 30, 30))])
def test_cg_on_chip_handles_side_by_side(large, small):
    systems = [cfm.varcoef_problem(s, 38) for s in (large, small)]
    handles = [cfm.CG(cfm.Stencil(k), cfm.CG_PERSISTENT, 12, 0.0) for k, _ in systems]
    for (k, f), h in zip(systems, handles):
        grid = (k.shape[-1], k.shape[-2], k.shape[0] if k.ndim == 3 else 1)
        xo, _, it_o, _, _ = oracle.krylov_stencil(k.ndim, grid, cfm.varcoef_coeffs(k), f, oracle.STD, 12, 0.0)
        x, st = h.solve(f.ravel())
        assert st.iterations == it_o
        np.testing.assert_array_equal(x, xo)


def grid_matrix(shape, values):
    """5-point CSR matrix of a grid: constant values (few row classes with equal values),
    or random symmetric ones (few classes of offsets only)."""
    ny, nx = shape
    rng = np.random.default_rng(34)
    we = np.ones((ny, nx)) if values == "constant" else rng.uniform(0.5, 1.5, (ny, nx))
    wn = np.ones((ny, nx)) if values == "constant" else rng.uniform(0.5, 1.5, (ny, nx))
    rowptr, col, val = [0], [], []
    for y in range(ny):
        for x in range(nx):
            i = y * nx + x
            ent = [(i, 8.0)]
            if x:
                ent.append((i - 1, -we[y, x - 1]))
            if x < nx - 1:
                ent.append((i + 1, -we[y, x]))
            if y:
                ent.append((i - nx, -wn[y - 1, x]))
            if y < ny - 1:
                ent.append((i + nx, -wn[y, x]))
            ent.sort()
            col += [c for c, _ in ent]
            val += [v for _, v in ent]
            rowptr.append(len(col))
    return np.array(rowptr, np.int32), np.array(col, np.int32), np.array(val)


def many_offsets_matrix(n):
    """Tridiagonal plus one symmetric far entry per row pair at growing distances: more
    than 256 kinds of rows, so no row classes."""
    far = {}
    for i in range(0, n // 2):
        j = n - 1 - i
        if j - i > 1:
            far[i], far[j] = j, i
    rowptr, col, val = [0], [], []
    for i in range(n):
        ent = {i: 8.0}
        if i:
            ent[i - 1] = -1.0
        if i < n - 1:
            ent[i + 1] = -1.0
        if i in far:
            ent[far[i]] = -0.5
        for c in sorted(ent):
            col.append(c)
            val.append(ent[c])
        rowptr.append(len(col))
    return np.array(rowptr, np.int32), np.array(col, np.int32), np.array(val)


@pytest.mark.parametrize("base", [0, 1])
@pytest.mark.parametrize("impl,method", [(cfm.CG_PERSISTENT, oracle.STD), (cfm.CG_DISCRETE, oracle.STD),
                                         (cfm.CG_PERSISTENT_PIPELINED, oracle.PIPELINED),
                                         (cfm.CG_MIXED, oracle.MIXED)])
@pytest.mark.parametrize("kind", ["constant", "variable", "many"])
def test_cg_row_classes(kind, impl, method, base):
    rowptr, col, val = many_offsets_matrix(1301) if kind == "many" else grid_matrix((61, 47), kind)
    b = cfm.uniform(35, len(rowptr) - 1)
    xo, st_o, it_o, rs_o, _ = oracle.krylov_csr(rowptr, col, val, b, method, 2000, 1e-8)
    A = cfm.CSR(rowptr + base, col + base, val)
    x, st = cfm.CG(A, impl, 2000, 1e-8).solve(b)
    assert st.status == st_o and st.iterations == it_o and st.refinements == rs_o
    np.testing.assert_array_equal(x, xo)


def class_limit_matrix(kind):
    """Matrices at the limits of the row classes: 256 kinds of rows and 257 (which only the
    offsets then group), rows of 32 entries and of 33 (no classes), an empty row."""
    n = 1300
    rows = [{i: 2.0} for i in range(n)]
    if kind.endswith("values"):
        for i in range(n):
            rows[i][i] = 2.0 + (i % 256) / 64
        if kind == "257 values":
            rows[n - 1][n - 1] = 7.0
    elif kind.endswith("entries"):
        for c in range(1, int(kind.split()[0])):
            rows[0][c] = rows[c][0] = -0.05
    else:
        for i in range(n - 1):
            rows[i][i + 1] = rows[i + 1][i] = -0.5
        for i in (699, 701):
            del rows[i][700]
        rows[700] = {}
    rowptr = np.cumsum([0] + [len(r) for r in rows]).astype(np.int32)
    col = np.array([c for r in rows for c in sorted(r)], np.int32)
    val = np.array([r[c] for r in rows for c in sorted(r)])
    b = cfm.uniform(48, n)
    b[700] = 0.0  # the empty row's equation
    return rowptr, col, val, b


@pytest.mark.parametrize("impl,method,maxiter,tol", [(cfm.CG_PERSISTENT, oracle.STD, 15, 0.0),
                                                     (cfm.CG_DISCRETE, oracle.STD, 15, 0.0),
                                                     (cfm.CG_PERSISTENT_PIPELINED, oracle.PIPELINED, 15, 0.0),
                                                     (cfm.CG_MIXED, oracle.MIXED, 2000, 1e-8)])
@pytest.mark.parametrize("kind", ["256 values", "257 values", "32 entries", "33 entries", "empty row"])
def test_cg_row_class_limits(kind, impl, method, maxiter, tol):
    rowptr, col, val, b = class_limit_matrix(kind)
    xo, st_o, it_o, rs_o, _ = oracle.krylov_csr(rowptr, col, val, b, method, maxiter, tol)
    x, st = cfm.CG(cfm.CSR(rowptr, col, val), impl, maxiter, tol).solve(b)
    assert st.status == st_o and st.iterations == it_o and st.refinements == rs_o
    np.testing.assert_array_equal(x, xo)


def test_cg_many_tiles_repeated():
    """More tiles than threads in a block (the sums behind a barrier), and a handle used
    again: the partials and flags of the first solve are still there."""
    n = 1100 * 1024 + 5
    rowptr, col, val = cfm.tridiag(n)
    A = cfm.CSR(rowptr, col, val)
    b = cfm.uniform(36, n)
    for impl, method in ((cfm.CG_PERSISTENT, oracle.STD), (cfm.CG_PERSISTENT_PIPELINED, oracle.PIPELINED)):
        h = cfm.CG(A, impl, 9, 0.0)
        xo, _, it_o, _, _ = oracle.krylov_csr(rowptr, col, val, b, method, 9, 0.0)
        for _ in range(3):
            x, st = h.solve(b)
            assert st.iterations == it_o
            np.testing.assert_array_equal(x, xo)


def test_batch_starting_plan_covers_every_system():
    """The plan a batch starts with (team sizes from 1 to 64 blocks side by side) solves
    every system to the same bits as one team size for all."""
    systems = [cfm.varcoef_problem(s, 40 + i) for i, s in
               enumerate([(300, 300), (16, 16), (64, 70), (40, 40, 40), (9, 9, 9), (128, 128), (33, 1), (200, 210)])]
    for prec in (cfm.FP64, cfm.FP32):
        B = cfm.Batch(systems)
        B.set_precision(prec)
        it0, st0, rr0, _ = B.solve()
        xs = [B.solution(i) for i in range(B.n)]
        assert (st0 == cfm.OK).all() and (rr0 <= 1e-8).all()
        B.set_plan([0], [4])
        it1, st1, _, _ = B.solve()
        assert (it0 == it1).all() and (st0 == st1).all()
        for i in range(B.n):
            np.testing.assert_array_equal(B.solution(i), xs[i])


# One tile, one tile and a remainder of two cells each way, fewer rows than a strip's four
# plus its halo, a remainder of half a tile in x.
@pytest.mark.parametrize("shape", [(32, 32), (34, 66), (6, 70), (68, 48)])
@pytest.mark.parametrize("m", [1, 3])
@pytest.mark.parametrize("mixed", [False, True])
def test_fpcg_smoothing_in_registers(shape, m, mixed):
    ny, nx = shape
    k, f = cfm.varcoef_problem(shape, 45)
    want, its, _, done = oracle.fpcg2d((nx, ny), cfm.varcoef_coeffs(k), f, 4, m, mixed)
    assert done == 1
    fp = cfm.FPCG(cfm.Stencil(k), k, None, maxiter=20000, tol=1e-8, smooth=4, truncation=m,
                  precision=cfm.FP32 if mixed else None)
    x, st = fp.solve(f)
    assert st.status == cfm.OK and st.iterations == its
    np.testing.assert_array_equal(x, want)


# stats.bytes counts the passes that the launched kernels make: a grid on chip is read and
# written once, the streaming kernel takes the first sweep alone and then up to eight per pass,
# the 3D kernel two, and the one-sweep kernels one.
@pytest.mark.parametrize("dims,shape,prec,impl,niter,passes", [
    (2, (200, 300), cfm.FP64, cfm.JACOBI_RESIDENT, 50, 1), (2, (200, 300), cfm.FP64, cfm.JACOBI_HOST_LOOP, 7, 7),
    (2, (2100, 2304), cfm.FP64, cfm.JACOBI_PERSISTENT, 17, 3), (3, (40, 39, 63), cfm.FP64, cfm.JACOBI_PERSISTENT, 10, 6),
    (3, (128, 128, 128), cfm.FP64, cfm.JACOBI_PERSISTENT, 10, 10)])
def test_jacobi_bytes_are_those_of_the_passes(dims, shape, prec, impl, niter, passes):
    with cfm.Jacobi(dims, shape[-1], shape[-2], shape[0] if dims == 3 else 1, prec, 1, impl) as j:
        st = j.run(niter)
        points = np.prod([n - 2 for n in shape])
        assert st.lups == points * niter
        assert st.bytes == points * passes * 2 * (8 if prec == cfm.FP64 else 4)


@pytest.mark.parametrize("kind,index,value", [("constant", lambda n, nnz: n, 0),
                                              ("variable", lambda n, nnz: n + 4 * (n + 1), 1),
                                              ("many", lambda n, nnz: 4 * nnz + 4 * (n + 1), 1)])
def test_cg_bytes_are_those_of_the_operator_form(kind, index, value):
    rowptr, col, val = many_offsets_matrix(1301) if kind == "many" else grid_matrix((61, 47), kind)
    n, nnz = len(rowptr) - 1, len(val)
    A = cfm.CSR(rowptr, col, val)
    for impl, word, vectors in ((cfm.CG_PERSISTENT, 8, 88), (cfm.CG_PERSISTENT_PIPELINED, 8, 96), (cfm.CG_MIXED, 4, 44)):
        st = cfm.CG(A, impl, 2000, 1e-8).solve(cfm.uniform(35, n))[1]
        assert st.bytes == st.iterations * (index(n, nnz) + value * word * nnz + vectors * n)


def test_cg_bytes_of_a_system_on_chip_do_not_grow_with_iterations():
    k, f = cfm.varcoef_problem((60, 70), 39)
    st = cfm.CG(cfm.Stencil(k), cfm.CG_PERSISTENT, 400, 1e-8).solve(f.ravel())[1]
    assert st.iterations > 50 and st.bytes == (3 * 8 + 16) * k.size
