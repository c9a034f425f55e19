"""The chain solver's forms (through the C ABI): the symmetric elimination
(Static steps without load stiffness) and the general one, each with an item
per thread for large levels and an item per warp for small ones; corners with
some DOFs fixed.  Every structure as the oracle solves it (1e-10 of the
coordinate scale, the same counts), and the same bits whatever form the size
of its batch selects."""
import numpy as np
import pytest

from giraffe_gb300 import configs, gpu
from giraffe_gb300.model import NodalLoad, Table
from oracle import oracle

pytestmark = pytest.mark.gpu


def chain(n, moment=False, fix=None, steps=3):
    s = configs.pipe_chain(n, 0.4, 0.03, [2e4, -1e4, 3e4], steps=steps, element_length=10.0 / n)
    if moment:
        s.loads.append(NodalLoad([2 * n], 0, Table(np.array([0.0, 1.0]), np.array([[0.0] * 6, [0, 0, 0, 2e3, 1e3, 5e2]]))))
    for node, mask in (fix or {}).items():
        s.clamp(node, mask)
    return s


def riser(n, pinned):
    s = configs.riser_chain(n, 0.4, 0.03, 1.0, 6.0, steps=4)
    if pinned:
        s.clamp(0, (1, 1, 1, 0, 0, 0))
    return s


def solve(structs):
    return gpu.solve(structs)


@pytest.mark.parametrize("make", [
    lambda: chain(1), lambda: chain(2), lambda: chain(3), lambda: chain(17), lambda: chain(33, moment=True),
    lambda: chain(1, moment=True), lambda: chain(2, moment=True),
    lambda: chain(20, fix={40: (0, 1, 0, 0, 0, 0)}), lambda: chain(21, fix={42: (1, 1, 1, 0, 0, 0), 20: (0, 0, 1, 0, 0, 0)}),
    lambda: chain(12, moment=True, fix={24: (1, 0, 0, 0, 0, 0), 12: (0, 1, 0, 0, 0, 0)}),
    lambda: riser(9, False), lambda: riser(10, True),
], ids=["1", "2", "3", "17", "33m", "1m", "2m", "roller", "pinned_and_guided", "fixed_m", "riser", "riser_pinned"])
def test_solves_as_the_oracle(gpu_ctx, make):
    s = make()
    finals, stats = solve([s])
    fo, so, _ = oracle.solve(s, 0)
    assert tuple(stats[0]) == tuple(so)
    scale = np.abs(fo[:, :3]).max()
    assert np.abs(finals[0][:, :3] - fo[:, :3]).max() <= 1e-10 * scale
    assert np.abs(finals[0][:, 6:] - fo[:, 6:]).max() <= 1e-9


@pytest.mark.parametrize("make", [lambda: chain(57), lambda: chain(57, moment=True), lambda: riser(57, True)],
                         ids=["symmetric", "general", "dynamic"])
def test_same_bits_in_a_batch_of_either_size(gpu_ctx, make):
    """One structure alone (every level below the thresholds), and among 260
    chains of 40 to 75 elements of both kinds (14,900 elements: the first
    levels above them)."""
    alone, _ = solve([make()])
    many = [chain(40 + i % 36, moment=i % 2 == 1, steps=1) for i in range(260)]
    batch, _ = solve(many[:100] + [make()] + many[100:])
    assert np.array_equal(alone[0], batch[100])
