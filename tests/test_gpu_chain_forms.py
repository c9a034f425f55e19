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


def chain(n, moment=None, fix=None, steps=3):
    """moment: node of a nodal moment (its stiffness is not symmetric), from the end if negative."""
    s = configs.pipe_chain(n, 0.4, 0.03, [2e4, -1e4, 3e4], steps=steps, element_length=10.0 / n)
    if moment is not None:
        s.loads.append(NodalLoad([moment % (2 * n + 1)], 0, Table(np.array([0.0, 1.0]), np.array([[0.0] * 6, [0, 0, 0, 2e3, 1e3, 5e2]]))))
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


CASES = {
    # the symmetric elimination: part counts around powers of two, moments and fixed DOFs at the ends
    "1": lambda: chain(1), "2": lambda: chain(2), "3": lambda: chain(3), "8": lambda: chain(8), "17": lambda: chain(17),
    "31": lambda: chain(31), "32": lambda: chain(32), "65": lambda: chain(65),
    "1_tip_moment": lambda: chain(1, -1), "33_tip_moment": lambda: chain(33, -1),
    "roller_tip": lambda: chain(20, fix={40: (0, 1, 0, 0, 0, 0)}),
    "pinned_tip_moment": lambda: chain(11, -1, fix={22: (1, 0, 1, 0, 0, 0)}),
    # the general one: moments or fixed DOFs inside the chain, Dynamic steps
    "2_moment": lambda: chain(2, 2), "3_midside_moment": lambda: chain(3, 3), "33_moment": lambda: chain(33, 20),
    "guided": lambda: chain(21, fix={42: (1, 1, 0, 0, 0, 0), 20: (0, 0, 1, 0, 0, 0)}),
    "guided_moment": lambda: chain(12, 8, fix={24: (1, 0, 0, 0, 0, 0), 12: (0, 1, 0, 0, 0, 0)}),
    "31_moment": lambda: chain(31, 6), "65_moment": lambda: chain(65, 64),
    "riser": lambda: riser(9, False), "riser_pinned": lambda: riser(10, True),
}


@pytest.mark.parametrize("make", CASES.values(), ids=CASES.keys())
def test_solves_as_the_oracle(gpu_ctx, make):
    s = make()
    finals, stats = solve([s])
    fo, so, _ = oracle.solve(s, 0)
    assert tuple(stats[0]) == tuple(so)
    scale = np.abs(fo[:, :3]).max()
    assert np.abs(finals[0][:, :3] - fo[:, :3]).max() <= 1e-10 * scale
    assert np.abs(finals[0][:, 6:] - fo[:, 6:]).max() <= 1e-9


@pytest.mark.parametrize("make", [lambda: chain(57), lambda: chain(57, -1), lambda: chain(57, 30), lambda: riser(57, True)],
                         ids=["symmetric", "tip_moment", "general", "dynamic"])
def test_same_bits_in_a_batch_of_either_size(gpu_ctx, make):
    """One structure alone (every level below the thresholds), and among 1,300
    chains of 40 to 75 elements of both kinds (37,000 elements of each: the
    first levels above them)."""
    alone, _ = solve([make()])
    many = [chain(40 + i % 36, 20 if i % 2 else None, steps=1) for i in range(1300)]
    batch, _ = solve(many[:100] + [make()] + many[100:])
    assert np.array_equal(alone[0], batch[100])
