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


# one tile, several, the row sweeps (the last grid also in the IEEE mode)
@pytest.mark.parametrize("ny,nx", [(2, 2), (9, 40), (65, 129), (1250, 1260)])
@pytest.mark.parametrize("arithmetic", ["exact", "fast"])
@pytest.mark.parametrize("ends", ["duration", "cap", "max_steps"])
@pytest.mark.parametrize("calm", [False, True])
def test_clock_advanced_by_the_step_equals_the_clock_kernel(ny, nx, arithmetic, ends, calm):
    """A run with a gauge has a clock kernel between two steps, one without
    advances the clock inside the second stage: the same steps, bits, number
    of steps and errors (the rough states of some sizes go non-finite)."""
    if ny > 1000 and ends != "duration":
        pytest.skip("covered by the smaller grids")
    z, U = _site(ny, nx, ny * 1000 + nx)
    if calm:
        U = torch.cat([torch.clamp(0.1 - z, min=0.0)[None], 0.01 * U[1:] * (z < 0.05)])
    cfg = SWEConfig(boundary_left="water_level", boundary_right="wall", boundary_top="wall", boundary_bottom="absorbing")
    kw = {"duration": {}, "cap": dict(max_dt_cap=4e-4), "max_steps": dict(max_steps=5)}[ends]
    out = []
    for gauges in ({}, {"g": (1, 1)}):
        m = SWE2D(z, torch.full_like(z, 0.02), 0.05, 0.07, config=cfg, train_dem=False, arithmetic=arithmetic)
        t = torch.linspace(0.0, 0.05, 33, device=DEV)
        m.set_dynamic_boundary(t, 0.1 + 0.05 * torch.sin(200.0 * t))
        m.gauge_indices, m.track_gauges = gauges, bool(gauges)
        with torch.no_grad():
            for t_end in (0.01, 0.05):  # the second finds another call's clock and level in the buffers
                try:
                    V, hmax = m(U[None], t_end=t_end, **kw)
                    out.append((m.last_forward_steps, V, hmax))
                except (FloatingPointError, RuntimeError) as err:
                    assert not calm or ends == "max_steps"
                    out.append((str(err),))
    for a, b in ((out[0], out[2]), (out[1], out[3])):
        assert a[0] == b[0]
        assert all(torch.equal(p, q) for p, q in zip(a[1:], b[1:]))


def test_clocked_step_refuses_a_shared_set():
    from diffswe2d_b200 import _native as nat
    z, U = _site(9, 40, 1)
    m = SWE2D(z, torch.full_like(z, 0.02), 0.5, 0.7, train_dem=False)
    buf = torch.zeros((4, 256), device=DEV)
    p = lambda k: nat.ptr(buf[k])  # noqa: E731
    args = [nat.ptr(U), nat.ptr(z), 1, nat.ptr(z), 1, 1, 9, 40, m._params(), p(0), 1, p(1), None, 0, 1, nat.ptr(U),
            p(2), nat.ptr(U), None]
    rc = nat.lib().swe_step_clocked_next_f32(*args, p(1), p(3), None, None, 0, None, nat.stream_handle(torch.device(DEV, 0)))
    assert rc == nat.SWE_EARG


@pytest.mark.parametrize("gauges", [{}, {"g": (1, 1)}])
def test_odd_chunks_give_the_steps_of_even_ones(gauges):
    z, U = _site(37, 53, 3)
    U = torch.cat([torch.clamp(0.1 - z, min=0.0)[None], 0.01 * U[1:] * (z < 0.05)])
    out = []
    for chunk in (32, 1, 3):
        m = SWE2D(z, torch.full_like(z, 0.02), 0.05, 0.07, train_dem=False)
        m.steps_per_chunk = chunk
        m.gauge_indices, m.track_gauges = gauges, bool(gauges)
        with torch.no_grad():
            V, hmax = m(U[None], t_end=0.1, boundary_level=0.1)
        out.append((m.last_forward_steps, list(m.ts_time), V, hmax))
    assert out[0][0] > 3
    for b in out[1:]:
        assert b[:2] == out[0][:2] and torch.equal(b[2], out[0][2]) and torch.equal(b[3], out[0][3])
