"""A Karhunen-Loeve perturbation of more columns than a launch has blocks in y
times the 128 columns that a block of its tables takes."""
import numpy as np
import pytest

from oracle import kl_oracle as ko

pytestmark = pytest.mark.gpu


def test_kl_of_a_wide_grid(gpu_ctx):
    from gpuocean_gb300.SWEsimulators.ModelErrorKL import ModelErrorKL
    from gpuocean_gb300.utils import Common
    nx, ny = 65535 * 128 + 5, 1
    stream = Common.Stream()
    me = ModelErrorKL(gpu_ctx, stream, nx, ny, 2000.0, 2500.0, Common.BoundaryConditions(), kl_decay=1.25,
                      kl_scaling=0.025, basis_x_start=1, basis_x_end=2, basis_y_start=1, basis_y_end=1)
    normals = np.array([[0.7, -1.1], [0.4, 0.9]], np.float32)
    eta = Common.CUDAArray2D(stream, nx, ny, 2, 2, np.zeros((ny + 4, nx + 4), np.float32))
    roll = (0.21, 0.43, 0.65, 0.87)
    me.perturbEta(eta, random_numbers=normals, perturbation_scale=0.7, roll_x_sin=roll[0], roll_y_sin=roll[1],
                  roll_x_cos=roll[2], roll_y_cos=roll[3])
    got = eta.download(stream)[2, 2:-2]
    want = ko.kl_d_eta(nx, ny, normals, 1, 2, 1, 1, True, True, np.float32(1.25), np.float32(0.025), 0.7, roll)[1, 1:-1]
    # the bar of the tables' test against the same oracle
    assert np.abs(got - want).max() <= 2e-5 * np.abs(want).max()
    eta.release()
    me.cleanUp()
