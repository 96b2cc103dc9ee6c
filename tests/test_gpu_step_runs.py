"""Runs of steady steps in one graph: any split of a rollout gives the same bits as single steps.

Runs begin once 288 steps were taken singly.
"""
import numpy as np
import pytest

from parallelspectralfluids3d_b200 import _lib as L
from parallelspectralfluids3d_b200.fixture import initial_coefficients, initial_particles
from parallelspectralfluids3d_b200.solver import Context

pytestmark = pytest.mark.gpu


def outcome(b, splits, particles):
    """State, particles and face velocities after every part of a rollout."""
    force = np.zeros(b.n_modes)
    force[0] = 2.0
    params = L.make_params(dt=0.01, viscosity=0.05, lifetime=9.0, flags=L.PSF_FLAG_RENORM | L.PSF_FLAG_FORCING, seed=4)
    out = []
    with Context(b, params, forcing=force) as ctx:
        ctx.set_state(initial_coefficients(b.n_modes, 1) * 20.0)
        if particles:
            p = initial_particles(b, 3001, 2)
            p[:, 3] = np.arange(3001) % 11  # respawns at every step: the tracer's step count shows
            ctx.set_particles(p)
        for part in splits:
            for n in part:
                ctx.step(n)
            out.append((ctx.get_state(), ctx.get_particles() if particles else None, ctx.get_velocity()))
    return out


@pytest.mark.parametrize("particles", [True, False])
@pytest.mark.parametrize("counts", [(314, 12, 11), (113, 225, 1, 24), (2, 336, 5, 17, 290, 330), (40, 400)])
def test_runs_equal_single_steps(small_bases, particles, counts):
    b = small_bases["sphere12x10x9"]
    whole = outcome(b, [[n] for n in counts], particles)
    single = outcome(b, [[1] * n for n in counts], particles)
    for a, c in zip(whole, single):
        for x, y in zip(a, c):
            assert x is None and y is None or np.array_equal(x, y)


def test_runs_after_changes(small_bases):
    """A change of state between runs restarts the pipeline; parameters drop the captured graphs."""
    b = small_bases["box576"]
    got = []
    for split in ([330, 16, 360], None):
        with Context(b, L.make_params(dt=0.01)) as ctx:
            ctx.set_particles(initial_particles(b, 500, 2))
            for k, n in enumerate([330, 16, 360]):
                if k == 2:
                    ctx.set_params(L.make_params(dt=0.02, integrator=L.PSF_RK1))
                else:
                    ctx.set_state(initial_coefficients(b.n_modes, k) * 10.0)
                for m in ([n] if split else [1] * n):
                    ctx.step(m)
            got.append((ctx.get_state(), ctx.get_particles()))
    assert all(np.array_equal(x, y) for x, y in zip(*got))
