"""Adaptive power-of-two block steps: a block with every particle on level 0 is exactly the
plain leapfrog step; levels follow the local dynamical time; energy is conserved."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(n, **kw):
    from blitzar_b200._lib import Engine
    kw.setdefault("physics_max_acceleration", 1e30)  # parity with the unclamped oracle
    return Engine(n, **kw)


def test_level_zero_blocks_equal_plain_leapfrog(gpu):
    from blitzar_b200 import ics

    n = 6000
    pos, vel, m = ics.plummer(n, seed=2)
    out = []
    for kw in (dict(), dict(adaptive_max_level=3, adaptive_eta=1e6)):
        with _engine(n, octree_theta=0.5, octree_softening=0.01, **kw) as e:
            e.set_state(pos, vel, m.astype(np.float32), f64=True)
            e.step(1e-3, 5)
            out.append(e.get_state(f64=True))
            if kw:
                assert (e.adaptive_levels() == 0).all()
                assert e.adaptive_updates() == 5 * n
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


def test_levels_follow_the_core(gpu):
    from blitzar_b200 import ics

    n = 20000
    pos, vel, m = ics.king(n, 4, 9.0)
    with _engine(n, octree_theta=0.5, octree_softening=0.01, adaptive_max_level=6, adaptive_eta=0.02) as e:
        e.set_state(pos, vel, m.astype(np.float32), f64=True)
        e.step(2e-3, 2)
        lv = e.adaptive_levels().astype(int)
        upd = e.adaptive_updates()
    r = np.linalg.norm(pos, axis=1)
    inner, outer = r < np.percentile(r, 10), r > np.percentile(r, 90)
    assert lv.min() >= 0 and lv.max() <= 6
    assert lv[inner].mean() > lv[outer].mean() + 0.5
    # every particle closes at least one step per block, the fine ones more
    assert upd >= 2 * n and upd > 2 * n * 1.2


def test_adaptive_energy_conservation(gpu):
    from blitzar_b200 import ics

    n = 16384
    pos, vel, m = ics.plummer(n, seed=6)
    with _engine(n, octree_theta=0.4, octree_softening=0.01, adaptive_max_level=5, adaptive_eta=0.02) as e:
        e.set_state(pos, vel, m.astype(np.float32), f64=True)
        k0, w0, _ = e.energy()
        e.step(8e-3, 25)
        k1, w1, _ = e.energy()
        lv = e.adaptive_levels()
    assert lv.max() >= 2  # the run did use several levels
    assert abs((k1 + w1) - (k0 + w0)) < 1e-3 * abs(k0 + w0)


@pytest.mark.parametrize("eta", [1e6, 0.02])
def test_counters_count_the_targets_evaluated(gpu, eta):
    """A block's last substep closes every particle, so its counters are a whole walk's: with one
    level (a fresh tree) those of a plain evaluation of the same positions; without a cutoff every
    listed pair is taken through the pair law."""
    from blitzar_b200 import ics

    n = 20_000
    pos, vel, m = ics.plummer(n, seed=9)
    with _engine(n, octree_theta=0.5, octree_softening=0.01, adaptive_max_level=5, adaptive_eta=eta) as e:
        e.set_state(pos, vel, m.astype(np.float32), f64=True)
        e.step(4e-3, 1)
        block = e.walk_counts()
        e.accelerations()
        plain = e.walk_counts()
    assert block[0] == block[1] and plain[0] == plain[1]
    if eta > 1:
        assert block == plain


def _direct(pos, mass, eps):
    d = pos[None] - pos[:, None]
    return ((mass[None] * ((d * d).sum(-1) + eps * eps) ** -1.5)[..., None] * d).sum(1)


def _level(a, v, eta, eps, dt, top):
    am, vm = np.linalg.norm(a, axis=1), np.linalg.norm(v, axis=1)
    stable = np.minimum(dt, np.minimum(eta * np.sqrt(eps / np.maximum(am, 1e-6)), eta * eps / np.maximum(vm, 1e-6)))
    return np.minimum(np.ceil(np.log2(dt / stable) - 1e-9).astype(int).clip(0), top)


def _block(pos, vel, mass, eps, dt, eta, top):
    """One block of hierarchical kick-drift-kick steps in FP64 with direct sums; returns the state and how
    often each particle closed a step."""
    acc = _direct(pos, mass, eps)
    level = _level(acc, vel, eta, eps, dt, top)
    L = int(level.max())
    closed = np.zeros(len(pos), int)
    for s in range(1 << L):
        opens = s % (1 << (L - level)) == 0
        vel = vel + np.where(opens[:, None], 0.5 * dt / (1 << level)[:, None] * acc, 0.0)
        pos = pos + dt / (1 << L) * vel
        closes = (s + 1) % (1 << (L - level)) == 0
        fresh = _direct(pos, mass, eps)
        acc = np.where(closes[:, None], fresh, acc)
        vel = vel + np.where(closes[:, None], 0.5 * dt / (1 << level)[:, None] * acc, 0.0)
        last = s + 1 == 1 << L
        coarsest = 0 if last else L - ((s + 1) & -(s + 1)).bit_length() + 1
        want = np.clip(_level(acc, vel, eta, eps, dt, top), coarsest, top if last else L)
        level = np.where(closes, want, level)
        closed += closes
    return pos, vel, closed


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("gsize", [1, 2, 5, 32])
def test_substeps_move_every_particle_as_direct_sums_do(gpu, order, gsize):
    """Substeps evaluate the closing members of a group, from one to all of them: with the opening angle
    near zero the block is that of FP64 direct sums, particle by particle, and closes as many steps."""
    from blitzar_b200 import ics

    n, eps, dt, eta, top = 900, 0.02, 8e-3, 0.05, 6
    pos, vel, m = ics.plummer(n, seed=21)
    mass = m.astype(np.float32)
    p, v, closed = _block(pos, vel, mass.astype(np.float64), eps, dt, eta, top)
    assert len(np.unique(closed)) >= 4  # several levels
    with _engine(n, octree_theta=1e-3, physics_min_theta=1e-3, octree_softening=eps, multipole_order=order,
                 walk_group_size=gsize, adaptive_max_level=top, adaptive_eta=eta) as e:
        e.set_state(pos, vel, mass, f64=True)
        e.step(dt, 1)
        gp, gv = e.get_state(f64=True)
        updates = e.adaptive_updates()
    kick = dt * np.linalg.norm(_direct(pos, mass.astype(np.float64), eps), axis=1)
    err = np.linalg.norm(gv - v, axis=1) / kick
    # FP32 sums of n terms; a particle whose level falls on the other side of the rule's comparison (none
    # of these seeds) would take other steps, one that was given another's force would be off by order 1
    assert err.max() < 1e-4, (err.max(), np.argmax(err))
    assert np.abs(gp - p).max() < 1e-4 * dt * kick.max()
    assert updates == closed.sum()
