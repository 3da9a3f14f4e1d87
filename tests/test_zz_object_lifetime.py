"""A mesh, an operator, a preconditioner and a solver made from one another are
destroyed children first and once each, whatever the order in which they are
closed: Python finalises the objects of a reference cycle in any order, and a
child's destructor uses its parent."""
import itertools

import pytest

from pdesolver_gb300 import eulergpu, problems


class FakeLibrary:
    """hands out numbers as handles and records what is destroyed"""

    def __init__(self):
        self.made = itertools.count(1)
        self.destroyed = []

    def __getattr__(self, name):
        def call(*args):
            if name.endswith("_create"):
                args[-1]._obj.value = next(self.made)
            elif name.endswith("_destroy"):
                self.destroyed.append(name)
            return 0
        return call


@pytest.mark.parametrize("order", list(itertools.permutations(range(4))))
def test_children_are_destroyed_before_their_parents(monkeypatch, order):
    lib = FakeLibrary()
    monkeypatch.setattr(eulergpu, "library", lambda: lib)
    ms, opts, _ = problems.config1(n=1, p=1, family="gamma", seed=1)
    g = eulergpu.GPUMesh(ms, opts)
    lo = eulergpu.LinearOperator(g)
    pc = eulergpu.BlockJacobiPC(lo)
    ls = eulergpu.LinearSolver(pc, lo)
    objects = (g, lo, pc, ls)
    for k in order:
        objects[k].close()
        objects[k].close()     # closing again changes nothing
    assert lib.destroyed == ["eg_ls_destroy", "eg_pc_destroy", "eg_lo_destroy", "eg_mesh_destroy"]
