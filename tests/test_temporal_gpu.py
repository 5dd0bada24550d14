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
