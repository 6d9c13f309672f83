"""The FP64 product of parity_march is no further from the exact product than that of the element-plane-pair kernel,
whose constants are the parity blocks' own entries."""
import numpy as np
import pytest
import torch

import voxel_b200 as vx

pytestmark = pytest.mark.gpu
CORNERS = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]


def exact(shape, ke, E, u):
    """K(E) u in extended precision."""
    nx, ny, nz = shape
    u = u.astype(np.longdouble).reshape(nx + 1, ny + 1, nz + 1, 3)
    ue = np.concatenate([u[i:i + nx, j:j + ny, k:k + nz] for i, j, k in CORNERS], axis=3)
    f = np.zeros_like(ue)
    for a in range(24):
        for b in range(24):
            f[..., a] += np.longdouble(ke[a, b]) * ue[..., b]
    f *= E.astype(np.longdouble).reshape(shape)[..., None]
    y = np.zeros_like(u)
    for n, (i, j, k) in enumerate(CORNERS):
        y[i:i + nx, j:j + ny, k:k + nz] += f[..., 3 * n:3 * n + 3]
    return y.reshape(-1)


def error(shape, ke, E, u, stream):
    op = vx.VoxelOperator(shape, ke, stream=stream)
    z = op.matvec(torch.as_tensor(u, device="cuda"), torch.as_tensor(E, device="cuda")).cpu().numpy()
    y = exact(shape, ke, E, u)
    return float(np.sqrt(((z - y) ** 2).sum() / (y ** 2).sum()))


# Integer elements: both kernels' constants are exact, so that only the roundings of the arithmetic are left.  Both
# make as many; the 2-norms of about 30,000 of them differ between two orders by chance by 1 / sqrt(30,000), and
# five times that, 3%, is allowed.
ELEMENTS = {"0.3": (vx.quadrature([1.0, 1.0, 1.0], 0.3), 1.0),
            "0.25 x 180": (np.rint(180 * vx.quadrature([1.0, 1.0, 1.0], 0.25)), 1.03),
            "0.3 x 1872": (np.rint(1872 * vx.quadrature([1.0, 1.0, 1.0], 0.3)), 1.03)}


@pytest.mark.parametrize("element", ELEMENTS)
@pytest.mark.parametrize("uniform", [False, True])
@pytest.mark.parametrize("shape", [(32, 16, 16), (20, 33, 17), (17, 48, 24)])
def test_fp64_product_error_is_at_most_the_pair_kernels(shape, uniform, element):
    rng = np.random.default_rng(3)
    ke, most = ELEMENTS[element]
    E = np.ones(int(np.prod(shape))) if uniform else 0.01 + 0.99 * rng.random(int(np.prod(shape))) ** 3
    u = rng.standard_normal(3 * vx.n_nodes(shape))
    march, xp = (error(shape, ke, E, u, stream) for stream in (None, "xp"))
    assert march <= most * xp, (march, xp)
