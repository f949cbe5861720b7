"""The IEEE stages in their two kernel forms, and the tile height that a
launch takes by itself, give the same bits: a batch large enough for the row
sweep against its members alone (shared-memory tiles)."""
import numpy as np
import pytest
import torch

from diffswe2d_b200 import SWE2D, SWEConfig

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _site(ny, nx, seed):
    rng = np.random.default_rng(seed)
    z = rng.uniform(-1.0, 0.2, (ny, nx)).astype(np.float32)
    h = np.maximum(rng.uniform(-0.3, 1.0, (ny, nx)), 0.0).astype(np.float32)
    U = np.stack([h, h * rng.uniform(-1, 1, h.shape), h * rng.uniform(-1, 1, h.shape)])
    return torch.from_numpy(z).to(DEV), torch.from_numpy(U.astype(np.float32)).to(DEV)


# batches just above 1.5 million cells: the sweep form
@pytest.mark.parametrize("ny,nx", [(2, 2), (9, 40), (37, 53), (65, 129), (244, 393)])
@pytest.mark.parametrize("friction", ["manning", "roughness_length"])
def test_sweep_and_tile_forms_agree(ny, nx, friction):
    z, U = _site(ny, nx, ny * 1000 + nx)
    B = min((3 << 19) // (ny * nx) + 1, 65535)
    cfg = SWEConfig(boundary_left="water_level", boundary_right="absorbing", boundary_top="wall",
                    boundary_bottom="transmissive", frictionmodel=friction)
    m = SWE2D(z, torch.full_like(z, 0.02), 0.5, 0.7, config=cfg, train_dem=False)
    one = U[None].contiguous()
    many = one.expand(B, -1, -1, -1).contiguous()
    with torch.no_grad():
        k = m.spatial_operator(one, boundary_level=0.1)
        ks = m.spatial_operator(many, boundary_level=0.1)
        V, dt = m.step(one, 0.0, 1.0, boundary_level=0.1)
        Vs, dts = m.step(many, 0.0, 1.0, boundary_level=0.1)
    assert dt == dts
    for b in (0, B // 2, B - 1):
        assert torch.equal(ks[b], k[0])
        assert torch.equal(Vs[b], V[0])


def test_bed_kernel_equals_the_bed_property():
    """Shared and batched beds, masked and NaN-free corrections, and the
    tanh-bounded form (which stays a PyTorch expression)."""
    g = torch.Generator().manual_seed(2)
    for shape, bound in (((1, 1, 7, 9), None), ((3, 1, 65, 129), None), ((1, 1, 7, 9), 0.5)):
        z = torch.rand(shape, generator=g).to(DEV)
        mask = (torch.rand(shape, generator=g) < 0.5).to(DEV)
        m = SWE2D(z, torch.full_like(z, 0.02), 0.5, 0.7, maximum_dem_correction=bound, valid_mask=mask)
        with torch.no_grad():
            m.dem_correction_parameter.copy_(torch.randn(shape, generator=g))
        assert torch.equal(m._bed_values(), m.bed.detach())
