"""The periodic mesh solve at the sides with the fused z transform and at those on each side of them,
against the same Green's function applied in FP64, by the potential and by its forces; the large sides
against cuFFT's 3-D FP32 transforms; and the tensor-core cutoff filter's pair counts against the FP64
distances."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [32, 64, 128, 256, 512])
@pytest.mark.parametrize("gradient,assign", [(0, 0), (2, 2)])
def test_potential_matches_fp64_solve(gpu, mesh, gradient, assign):
    from blitzar_b200._lib import Engine

    rng = np.random.default_rng(mesh)
    n, rs = 20_000, 1.1
    with Engine(n, solver=1, box_length=1.0, treepm_grid_size=mesh, treepm_r_split_cells=rs, treepm_assignment=assign,
                treepm_gradient=gradient, treepm_window_floor=0.08) as e:
        e.set_state(rng.random((n, 3)), None, ((rng.random(n) + 0.5) / n).astype(np.float32), f64=True)
        rho = e.pm_mesh(0).reshape(mesh, mesh, mesh).astype(np.float64)
        phi = e.pm_mesh(1).reshape(mesh, mesh, mesh)
    k = 2 * np.pi * np.fft.fftfreq(mesh, 1 / mesh)
    kr = 2 * np.pi * np.fft.rfftfreq(mesh, 1 / mesh)
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kr[None, None, :] ** 2
    s, sr = np.sinc(k / (2 * np.pi * mesh)), np.sinc(kr / (2 * np.pi * mesh))
    window = (s[:, None, None] * s[None, :, None] * sr[None, None, :]) ** (2 * (assign + 2))
    k2[0, 0, 0] = 1.0
    green = 4 * np.pi * np.exp(-k2 * (rs / mesh) ** 2) / (k2 * np.maximum(window, 0.08))
    green[0, 0, 0] = 0.0
    ref = np.fft.irfftn(np.fft.rfftn(rho) * green, s=rho.shape, axes=(0, 1, 2))
    # two FP32 transforms of M^3 points: a few 2^-24 sqrt(log2 M^3) of the norm, far below 2e-6
    assert np.linalg.norm(phi - ref) < 2e-6 * np.linalg.norm(ref)


def _lattice_solve(mesh, gradient, assign):
    """Density and potential meshes of a displaced lattice of half the side, and the Green's function
    of the solve in FP64, on the GPU.  2^k particles of mass 2^-k at eighths of a cell: the sums of a CIC
    deposit are exact, so it repeats whatever the order of its atomics."""
    import torch

    from blitzar_b200 import ics
    from blitzar_b200._lib import Engine

    rs = 0.95
    pos, _, m = ics.grf_grid(mesh // 2, seed=mesh)
    pos = np.rint(pos * (8 * mesh)) / (8 * mesh) % 1.0
    with Engine(len(m), solver=1, box_length=1.0, treepm_grid_size=mesh, treepm_r_split_cells=rs,
                treepm_assignment=assign, treepm_gradient=gradient, treepm_window_floor=0.08) as e:
        e.set_state(pos, None, m.astype(np.float32), f64=True)
        rho, phi = (torch.from_numpy(e.pm_mesh(w)).cuda().reshape(1, mesh, mesh, mesh) for w in (0, 1))
    k = 2 * np.pi * torch.fft.fftfreq(mesh, 1 / mesh, dtype=torch.float64, device="cuda")
    kr = 2 * np.pi * torch.fft.rfftfreq(mesh, 1 / mesh, dtype=torch.float64, device="cuda")
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kr[None, None, :] ** 2
    s, sr = torch.sinc(k / (2 * np.pi * mesh)), torch.sinc(kr / (2 * np.pi * mesh))
    window = (s[:, None, None] * s[None, :, None] * sr[None, None, :]) ** (2 * (assign + 2))
    k2[0, 0, 0] = 1.0
    green = 4 * np.pi * torch.exp(-k2 * (rs / mesh) ** 2) / (k2 * window.clamp_min(0.08))
    green[0, 0, 0] = 0.0
    return rho, phi, green


def _force_difference(a, b):
    """2-norm of the difference of two potentials' centred differences over that of b's."""
    num = den = 0.0
    for axis in (1, 2, 3):
        d = [(f.roll(-1, axis) - f.roll(1, axis)).double() for f in (a.double(), b.double())]
        num += float(((d[0] - d[1]) ** 2).sum())
        den += float((d[1] ** 2).sum())
    return (num / den) ** 0.5


@pytest.mark.parametrize("mesh", [64, 128, 256, 512])
@pytest.mark.parametrize("gradient,assign", [(0, 0), (2, 2)])
def test_mesh_forces_match_fp64_solve(gpu, mesh, gradient, assign):
    """The potential's FP32 rounding, a few 2^-24 of its norm, which the longest waves fill, divided by
    the cell: of the order of 2^-24 (6e-8) / pi of the force times the side, whatever the transforms."""
    import torch

    rho, phi, green = _lattice_solve(mesh, gradient, assign)
    ref = torch.fft.irfftn(torch.fft.rfftn(rho.double(), dim=(1, 2, 3)) * green, s=(mesh,) * 3, dim=(1, 2, 3))
    assert _force_difference(phi, ref) < 2 * 2.0 ** -24 / np.pi * mesh


@pytest.mark.parametrize("mesh", [256, 512])
@pytest.mark.parametrize("gradient", [0, 2])
def test_large_sides_round_as_the_3d_transforms(gpu, mesh, gradient):
    """Sides of 256 and more give cuFFT's 3-D FP32 solve, rounding included.  torch's (the batch axis
    has it plan all three axes at once) shares the forward rounding bit for bit; a table entry an FP32
    unit away redraws part of the inverse's: 0.4 to 0.6e-8 of the force times the side.  A solve by
    other transforms lies 1.5 to 1.7e-8 away."""
    import torch

    rho, phi, green = _lattice_solve(mesh, gradient, 0)
    spec = torch.fft.rfftn(rho, dim=(1, 2, 3)) * green.float()
    ref = torch.fft.irfftn(spec, s=(mesh,) * 3, dim=(1, 2, 3))
    assert _force_difference(phi, ref) < 1e-8 * mesh


def _pairs_box(side, shift, seed):
    """Jittered lattice of close pairs: no octree leaf (at 16 a leaf) holds a single particle, which
    the walk would take as a point mass and not as a pair."""
    rng = np.random.default_rng(seed)
    g = (np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) / side
    p = g + 0.2 / side * rng.standard_normal(g.shape) + shift
    pos = (np.concatenate([p, p + 1e-4 / side * rng.standard_normal(g.shape)]) % 1.0).astype(np.float32)
    pos[pos >= 1.0] = 0.0
    return pos


@pytest.mark.parametrize("rcf", [0.3, 4.5, 5.0])
@pytest.mark.parametrize("side,shift,seed", [(16, 0.0, 1), (12, 0.4999, 1), (21, 0.3, 2)])
def test_cutoff_filter_counts_every_pair(gpu, rcf, side, shift, seed):
    """Pairs through the pair law of a walk that only filters = pairs inside the cutoff, whether the
    group is far wider than the cutoff (scalar filter) or not; FP64 distances of the FP32 positions,
    pairs within 2e-6 of the cutoff (rounding of a periodic image) left open."""
    from scipy.spatial import cKDTree

    from blitzar_b200._lib import Engine

    pos = _pairs_box(side, shift, seed)
    n = len(pos)
    with Engine(n, solver=1, box_length=1.0, treepm_grid_size=64, treepm_r_split_cells=1.0, treepm_r_cut_factor=rcf,
                treepm_gradient=2, treepm_assignment=2, treepm_window_floor=0.0, treepm_node_size_factor=1e-6,
                multipole_order=1, octree_softening=0.02 / side) as e:
        e.set_state(pos, None, np.full(n, 1.0 / n, np.float32))
        e.accelerations()
        _, evaluated, nodes = e.walk_counts()
    assert nodes == 0
    tree = cKDTree(pos.astype(np.float64), boxsize=1.0)
    lo, hi = (tree.count_neighbors(tree, rcf / 64 * f) for f in (1 - 2e-6, 1 + 2e-6))
    assert lo <= evaluated <= hi, (lo, evaluated, hi)
