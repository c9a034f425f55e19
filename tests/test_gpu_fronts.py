"""The multifrontal LU of Shell_1 structures (through the C ABI) where its
schedule has edges: single elements and single fronts, fronts on either side
of the shared-memory limit, meshes of several components, strips, nodes with
load stiffness, and structures of different heights in one batch.  Each
structure as the oracle's banded LU with partial pivoting solves it: the same
step counts and 1e-10 of the coordinate scale (the plain path's stated
tolerance)."""
import numpy as np
import pytest

from giraffe_gb300 import configs, gpu
from giraffe_gb300.model import NodalLoad, Table
from oracle import oracle

pytestmark = pytest.mark.gpu


def strip(nx, ny, steps=3):
    """nx x ny squares of the plate family, clamped along every edge but one long one."""
    s = configs.square_plate(max(nx, ny), steps=steps)
    m = 2 * max(nx, ny) + 1
    keep = [i for i in range(m * m) if i % m <= 2 * nx and i // m <= 2 * ny]
    new = {old: k for k, old in enumerate(keep)}
    shells = [tuple(new[q] for q in row[:6]) + tuple(row[6:]) for row in s.shells if all(q in new for q in row[:6])]
    s.shells = shells
    s.nodes = s.nodes[keep]
    s.constraints = np.zeros((len(keep), 6), dtype=np.int32)
    for k, old in enumerate(keep):
        if old % m in (0, 2 * nx) or old // m == 0:
            s.constraints[k] = 1
    s.loads[0].shells = list(range(len(shells)))
    return s


def two_plates(n1, n2):
    """Two plates apart in one structure: the graph has two components."""
    a, b = configs.square_plate(n1, steps=3), configs.square_plate(n2, steps=3)
    k = a.n_nodes
    a.nodes = np.concatenate([a.nodes, b.nodes + [3.0, 0.0, 0.0]])
    a.shells.extend([tuple(q + k for q in row[:6]) + tuple(row[6:]) for row in b.shells])
    a.constraints = np.concatenate([a.constraints, b.constraints])
    a.loads[0].shells = list(range(len(a.shells)))
    return a


def loaded(n):
    """A plate with a moment on a midside node: load stiffness in K_AA."""
    s = configs.square_plate(n, steps=3)
    m = 2 * n + 1
    node = 2 * (n // 2) * m + 2 * (n // 2) + 1
    s.loads.append(NodalLoad([node], 0, Table(np.array([0.0, 1.0]), np.array([[0.0] * 6, [0, 0, -200.0, 15.0, 5.0, 0]]))))
    return s


@pytest.mark.parametrize("make", [
    lambda: configs.square_plate(1, steps=2), lambda: configs.square_plate(2, steps=2),
    lambda: configs.square_plate(3, steps=2), lambda: configs.square_plate(5, steps=2),
    lambda: configs.square_plate(13, steps=2), lambda: strip(1, 1), lambda: strip(9, 1), lambda: strip(12, 3),
    lambda: two_plates(2, 5), lambda: loaded(4), lambda: loaded(9),
], ids=["plate1", "plate2", "plate3", "plate5", "plate13", "strip1x1", "strip9x1", "strip12x3", "two", "loaded4", "loaded9"])
def test_solves_as_the_oracle(gpu_ctx, make):
    s = make()
    b = gpu.BatchSolver(gpu_ctx, [s, configs.square_plate(4, steps=2), make()])
    b.reset()
    b.run()
    finals, stats = b.results()
    b.close()
    fo, so, _ = oracle.solve(s, 0)
    assert tuple(stats[0]) == tuple(so)
    scale = np.abs(fo[:, :3]).max()
    assert np.abs(finals[0][:, :3] - fo[:, :3]).max() <= 1e-10 * scale
    assert np.abs(finals[0][:, 6:] - fo[:, 6:]).max() <= 1e-9
    # the same structure elsewhere in the batch, and alone: the same bits
    assert np.array_equal(finals[0], finals[2])
    alone, _ = gpu.solve([make()])
    assert np.array_equal(finals[0], alone[0])
