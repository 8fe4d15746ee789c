"""Copies of meshes and projections: the attribute-wise deep copy builds what
copy.deepcopy's own walk builds (aliases and extra attributes included), and a
projection's vector follows its cells however their values are changed."""
import copy
import pickle

import numpy as np
import pytest

from rtg import workloads as W
from rtg.mesh import Mesh
from rtg.projection import Projection


class _SubMesh(Mesh):
    pass


def _shape(x):
    """Types, values and aliases reachable from x, in order."""
    seen, out = {}, []

    def walk(o):
        if isinstance(o, np.ndarray):
            out.append(o.tolist())
        elif isinstance(o, (list, dict, tuple)) or hasattr(o, "__dict__"):
            if id(o) in seen:
                out.append(seen[id(o)])
                return
            seen[id(o)] = len(seen)
            out.append(type(o).__name__)
            for v in (list(o.items()) if isinstance(o, dict) else o if isinstance(o, (list, tuple)) else [o.__dict__]):
                walk(v)
        else:
            out.append(o)

    walk(x)
    return out


@pytest.mark.parametrize("extras", [False, True])
def test_copy_equals_the_generic_walk(extras):
    m = W.small_random_mesh()
    if extras:
        col = m.cols[sorted(m.cols)[0]]
        m.extra, m.me, m.arr = {"a": [col, (1, [2])], 3: col.ndofs}, m, np.arange(3)
    c = copy.deepcopy(m)
    ref = pickle.loads(pickle.dumps(m))
    assert _shape(c) == _shape(ref) == _shape(m) and c == m
    k = sorted(m.cols)[0]
    c.cols[k].ndofs[0] += 1
    assert c != m and m == ref
    s = _SubMesh([1., 1.], [False, False], [2, 2, 2], True)
    s.q = [1]
    t = copy.deepcopy(s)
    assert type(t) is _SubMesh and t == s and t.q == [1] and t.q is not s.q


@pytest.mark.parametrize("make", [lambda p: p, copy.deepcopy, copy.copy, lambda p: pickle.loads(pickle.dumps(p))])
def test_vector_follows_the_cells(make):
    m = W.small_random_mesh()
    p = make(Projection(m, lambda x, y, th: x + 2. * y + th))
    v = p.to_vector()
    k = sorted(p.cols)[1]
    kk = sorted(p.cols[k].cells)[0]
    cells = p.cols[k].cells
    at = sum(c.vals.size for c in p.cols[sorted(p.cols)[0]].cells.values())
    cells[kk].vals[0, 0, 0] = 9.
    v[at] = 9.
    np.testing.assert_array_equal(p.to_vector(), v)
    cells[kk].vals = cells[kk].vals + 1.
    n = cells[kk].vals.size
    v[at:at + n] += 1.
    np.testing.assert_array_equal(p.to_vector(), v)
    w = p.to_vector()
    w[:] = 0.
    np.testing.assert_array_equal(p.to_vector(), v)
    q = Projection(m).from_vector(v)
    assert q.from_vector(np.concatenate([v, [5.]])).to_vector().tolist() == v.tolist()
    v[0] = 4.
    assert q.to_vector()[0] != 4.


def test_subclasses_are_copied_as_they_say():
    """Wherever a subclass is defined (here: one that names the package's module as its own): state outside of the
    attributes is copied, and a __deepcopy__ of its own or of another base is taken."""
    class Slotted(Mesh):
        __slots__ = ("kept",)

    Slotted.__module__ = Mesh.__module__
    s = Slotted([1., 1.], [False, False], [2, 2, 2], True)
    s.kept, s.q = [1], [2]
    t = copy.deepcopy(s)
    assert type(t) is Slotted and t == s
    assert t.kept == [1] and t.kept is not s.kept and t.q == [2] and t.q is not s.q

    class Own:
        def __deepcopy__(self, memo):
            return "own"

    class First(Own, Mesh):
        pass

    class Last(Slotted, Own):
        pass

    for cls in (First, Last):
        assert copy.deepcopy(cls([1., 1.], [False, False], [2, 2, 2], True)) == "own"
