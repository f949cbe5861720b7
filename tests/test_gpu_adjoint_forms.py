"""The forms of the step adjoint against one another: of a single step (level
sides face by face, the predictor given) and of a run's steps (the predictor
made from U and k1), at grids where tiles of 32 x 16 cells can go wrong, with
zero, wild and NaN cotangents and with buffers shared."""
import pytest
import torch

from diffswe2d_b200 import SWE2D, SWEConfig
from diffswe2d_b200.adjoint import AdjointStepper

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SIDES = {"level": ("water_level", "wall", "absorbing", "transmissive"), "periodic": ("periodic",) * 4,
         "walls": ("wall",) * 4}
# all frame, one tile less one, exactly one, one and a cell, several
GRIDS = [(2, 2), (3, 5), (5, 4), (15, 31), (16, 32), (17, 33), (50, 67)]


def _problem(B, ny, nx, sides, arithmetic="exact", dry=0.15):
    g = torch.Generator().manual_seed(ny * 100 + nx + B)
    z = torch.rand((B, 1, ny, nx), generator=g) * 0.3 - 0.2
    h = torch.clamp(torch.rand((B, 1, ny, nx), generator=g) * 0.6 - dry, min=0.0)
    U = torch.cat([h, h * torch.randn((B, 2, ny, nx), generator=g)], 1).to(DEV)
    lam = torch.randn(U.shape, generator=g).to(DEV)
    z = z.to(DEV)
    cfg = SWEConfig(**dict(zip(("boundary_left", "boundary_right", "boundary_top", "boundary_bottom"), SIDES[sides])))
    m = SWE2D(z, torch.full_like(z, 0.02), 0.5, 0.7, config=cfg, train_dem=False, arithmetic=arithmetic)
    return m, U, lam, torch.linspace(0.05, 0.15, B, device=DEV)


def _stepper(m, U, run, bed_grad=True):
    B, _, ny, nx = U.shape
    return AdjointStepper(m, B, ny, nx, torch.device(DEV), B, bed_grad=bed_grad, run=run)


def _stages(m, U, level, dt):
    """k1, the predictor and k2 of a step."""
    st = _stepper(m, U, False, False)
    k1, P, k2 = (torch.empty_like(U) for _ in range(3))
    st._tendency(U, level, k1)
    st._pointwise(2, U, k1, dt, None, None, None, P)
    st._tendency(P, level, k2)
    return k1, P, k2


def _adjoint(m, U, lam, level, dt, run, stages):
    """Adjoints of the input state, the roughness and the bed of one step,
    and of the level per member."""
    k1, _, k2 = stages
    st = _stepper(m, U, run)
    lam_U, lam_n = torch.empty_like(U), torch.zeros_like(st.n)
    part = st(U, level, dt, lam.contiguous(), lam_U, lam_n, K1=k1, K2=k2, overwrite=True)
    return lam_U, lam_n, st.lam_bed, part.reshape(2, U.shape[0], -1).sum(dim=(0, 2))


@pytest.mark.parametrize("ny,nx", GRIDS)
@pytest.mark.parametrize("arithmetic", ["exact", "fast"])
@pytest.mark.parametrize("sides", sorted(SIDES))
def test_stage2_of_a_run_equals_that_of_a_single_step(ny, nx, arithmetic, sides):
    """swe_adj_stage2_k1_f32 against mode 2 of swe_adj_pointwise_f32 and
    swe_adj_stage2_f32.  Without level sides the IEEE forms evaluate the same
    operations on the same predictor: the same bits.  Else, along level
    sides, sums in another order (a few dozen roundings: 1e-5 normwise; the
    tolerance mode's approximations: 1e-4)."""
    m, U, lam, level = _problem(2, ny, nx, sides, arithmetic)
    k1, P, _ = _stages(m, U, level, 0.01)
    out = []
    for run in (False, True):
        st, lam_U = _stepper(m, U, run), torch.ones_like(U)
        st.lam_k.copy_(lam)
        st._stage2(P, U, k1, level, 0.01, lam_U)
        out.append((lam_U, st.lam_k1, st.lam_bed, st.part[0].reshape(2, -1).sum(1)))
    bound = 1e-5 if arithmetic == "exact" else 1e-4
    scale = float(torch.cat([q.reshape(-1) for q in out[0][:2]]).abs().max())
    for a, b in zip(*out):
        assert float((a - b).abs().max()) <= bound * max(scale, float(a.abs().max()))
        assert sides == "level" or arithmetic == "fast" or torch.equal(a, b)
    if sides == "level" and arithmetic == "exact" and min(ny, nx) > 4:
        for k in range(3):  # further than two cells from the sides: the same bits
            assert torch.equal(out[0][k][..., 2:-2, 2:-2], out[1][k][..., 2:-2, 2:-2])


@pytest.mark.parametrize("run", [False, True])
@pytest.mark.parametrize("arithmetic", ["exact", "fast"])
def test_step_adjoint_of_different_patches_per_member(run, arithmetic):
    """Cotangents that are zero outside a patch, another one per member (one
    has none): exactly zero beyond the reach of a step, the dense cotangents'
    bits well inside."""
    ny, nx, reach = 67, 101, 4
    m, U, lam, level = _problem(4, ny, nx, "level", arithmetic)
    mask = torch.zeros((4, 1, ny, nx), device=DEV)
    for b, (j0, j1, i0, i1) in enumerate([(20, 36, 30, 60), (0, 0, 0, 0), (40, 67, 60, 101), (0, 18, 0, 40)]):
        mask[b, :, j0:j1, i0:i1] = 1.0
    grow = lambda q: torch.nn.functional.max_pool2d(q, 2 * reach + 1, 1, reach)  # noqa: E731
    far, inner = grow(mask) == 0, grow(1.0 - mask) == 0
    stages = _stages(m, U, level, 0.01)
    full, part = (_adjoint(m, U, q, level, 0.01, run, stages) for q in (lam, lam * mask))
    for a, b in zip(full[:3], part[:3]):
        a, b = a.reshape(4, -1, ny, nx), b.reshape(4, -1, ny, nx)
        assert bool((b[far.expand_as(b)] == 0.0).all())
        assert torch.equal(a[inner.expand_as(a)], b[inner.expand_as(b)])
    assert float(part[3][1]) == 0.0 and float(part[3][3]) != 0.0


@pytest.mark.parametrize("run", [False, True])
@pytest.mark.parametrize("what", ["nan cotangent", "deep cell", "fast cell"])
def test_step_adjoint_around_a_wild_cell(run, what):
    """A NaN cotangent, or a cell deeper or faster than the zero skips
    accept, in a tile of zeros: further away than a step reaches, what other
    cells give does not change by a bit, and is zero where it was."""
    ny, nx, reach = 67, 101, 5
    m, U, lam, level = _problem(1, ny, nx, "walls", dry=-0.2)
    lam[..., :40] = 0.0
    V, mu = U.clone(), lam.clone()
    if what == "nan cotangent":
        mu[0, 1, 30, 15] = float("nan")
    elif what == "deep cell":
        V[0, 0, 30, 15] = 5e8
    else:
        V[0, 1, 30, 15] = 3e9 * V[0, 0, 30, 15]
    dt = 1e-13
    a = _adjoint(m, U, lam, level, dt, run, _stages(m, U, level, dt))
    b = _adjoint(m, V, mu, level, dt, run, _stages(m, V, level, dt))
    far = torch.ones((ny, nx), dtype=torch.bool, device=DEV)
    far[30 - reach:31 + reach, 15 - reach:16 + reach] = False
    for p, q in zip(a[:3], b[:3]):
        assert torch.equal(p.reshape(-1, ny, nx)[:, far], q.reshape(-1, ny, nx)[:, far])
        assert bool((p.reshape(-1, ny, nx)[:, :, :36] == 0).all())
    assert what != "nan cotangent" or bool(b[0][0, :, 30, 15].isnan().any())


@pytest.mark.parametrize("run", [False, True])
@pytest.mark.parametrize("ny,nx", [(5, 4), (20, 25), (50, 67)])
def test_stage2_writes_over_its_own_cotangent(run, ny, nx):
    """lam_k1 may be the lam_k2 buffer (with 3 B ny nx more floats of scratch)."""
    m, U, lam, level = _problem(3, ny, nx, "level")
    k1, P, _ = _stages(m, U, level, 0.01)
    out = []
    for shared in (False, True):
        st, lam_U = _stepper(m, U, run), torch.ones_like(U)
        st.cx = torch.full((st.cx.numel() + U.numel(),), float("nan"), device=DEV)
        st.lam_k.copy_(lam)
        if shared:
            st.lam_k1 = st.lam_k
        st._stage2(P, U, k1, level, 0.01, lam_U)
        out.append((lam_U, st.lam_k1, st.lam_bed, st.part[0]))
    for a, b in zip(*out):
        assert torch.equal(a, b) and not bool(a.isnan().any())


@pytest.mark.parametrize("arithmetic", ["exact", "fast"])
def test_forward_with_a_level_per_member(arithmetic):
    """The device loop, whose second stage advances the clock, against the
    host loop (forced by a callback)."""
    m, U, _, level = _problem(3, 37, 53, "level", arithmetic)
    z = m.bed.detach()
    U = torch.cat([torch.clamp(0.1 - z, min=0.0), 0.01 * U[:, 1:] * (z < 0.05)], 1)  # calm water
    with torch.no_grad():
        V, hmax = m(U, t_end=1.5, boundary_level=level)
        steps = m.last_forward_steps
        W, hm = m(U, t_end=1.5, boundary_level=level, callback=lambda *a: None)
    assert steps == m.last_forward_steps and steps > 3
    assert torch.equal(V, W) and torch.equal(hmax, hm)


@pytest.mark.parametrize("ny,nx", [(20, 25), (50, 67)])
def test_a_chunk_of_one_step_is_a_single_step(ny, nx):
    """forward_checkpointed over one step gives the gradients of step(), the
    level's included, bit for bit."""
    from diffswe2d_b200.adjoint import forward_checkpointed
    m, U, lam, level = _problem(8, ny, nx, "level")
    grads = []
    for chunk in (False, True):
        V, lv = U.clone().requires_grad_(True), level.clone().requires_grad_(True)
        if chunk:
            W = forward_checkpointed(m, V, 1e-3, boundary_level=lv)
            assert m.last_forward_steps == 1
        else:
            W, dt = m.step(V, 0.0, 1e-3, boundary_level=lv)
        (W * lam).sum().backward()
        grads.append((W.detach(), V.grad, lv.grad))
    for a, b in zip(*grads):
        assert torch.equal(a, b)
