"""Nodal function on the hp mesh: the solution container returned by solve.

Mirrors dg/projection/class_Projection.py:17-97: ``Projection(mesh, func)``
samples func(x, y, th) at the nodes; ``cols[col_key].cells[cell_key].vals`` is
an [nx, ny, nth] array; ``to_vector``/``from_vector`` use the global DOF order
(dg/projection/to_vector.py:11-44, from_vector.py:11-40); ``to_file`` writes the
vector as raw float64 plus the mesh JSON (dg/projection/to_file.py:10-19)."""

import copy
import operator

import numpy as np

from .layout import MeshLayout, _eval
from . import mesh as _mesh


class ProjectionCell:
    def __init__(self, cell, vals):
        self.pos = cell.pos
        self.idx = cell.idx
        self.lv = cell.lv
        self.key = cell.key
        self.is_lf = cell.is_lf
        self.ndofs = cell.ndofs
        self.quadrant = cell.quadrant
        self.vals = vals

    def __eq__(self, other):
        return (self.key == other.key and self.ndofs == other.ndofs
                and np.array_equal(self.vals, other.vals))


class ProjectionColumn:
    def __init__(self, col, cells):
        self.pos = col.pos
        self.idx = col.idx
        self.lv = col.lv
        self.key = col.key
        self.is_lf = col.is_lf
        self.ndofs = col.ndofs
        self.nhbr_keys = col.nhbr_keys
        self.cells = cells

    def __eq__(self, other):
        return self.key == other.key and self.cells == other.cells


class Projection:
    def __init__(self, mesh, func=None):
        self._set_mesh(mesh)
        lay = MeshLayout(self.mesh)
        if func is None:
            vec = np.zeros(lay.N)
        else:
            X, Y, T = lay.node_coords()
            if self.mesh.has_th:
                vec = np.array(_eval(func, X, Y, T), dtype=np.float64)
            else:
                vec = np.array(_eval(lambda x, y, th: func(x, y), X, Y, T), dtype=np.float64)
        self._build(lay, vec)

    @classmethod
    def _of_vector(cls, mesh, vec):
        """Projection(mesh).from_vector(vec), built once"""
        self = cls.__new__(cls)
        self._set_mesh(mesh)
        return self.from_vector(vec)

    def _set_mesh(self, mesh):
        self.mesh = copy.deepcopy(mesh)
        self.Ls = self.mesh.Ls
        self.pbcs = self.mesh.pbcs
        self.has_th = self.mesh.has_th

    def _build(self, lay, vec):
        """The cells' values are views of one vector in global order."""
        vec = np.array(vec[:lay.N], order="C")
        start, off = lay.col_elem_start.tolist(), lay.elem_off.tolist()
        self.cols = {}
        views = []
        for ci, ck in enumerate(lay.col_keys):
            col = self.mesh.cols[ck]
            nx, ny = col.ndofs[0], col.ndofs[1]
            cells = {}
            for e in range(start[ci], start[ci + 1]):
                kk = lay.elem_keys[e][1]
                cell = col.cells[kk]
                vals = vec[off[e]:off[e + 1]].reshape(nx, ny, cell.ndofs[0])
                views.append(vals)
                cells[kk] = ProjectionCell(cell, vals)
            self.cols[ck] = ProjectionColumn(col, cells)
        self._flat = (vec, views)

    def __getstate__(self):
        """Copies and pickles hold the cells' values, not the vector besides."""
        state = self.__dict__.copy()
        state.pop("_flat", None)
        return state

    def to_vector(self):
        out = []
        for ck in sorted(self.cols.keys()):
            cells = self.cols[ck].cells
            out += [cells[kk].vals for kk in sorted(cells.keys())]
        # as built: every cell still holds its own view of the vector
        vec, views = self.__dict__.get("_flat", (None, ()))
        if len(out) == len(views) and all(map(operator.is_, out, views)) and all(v.base is vec for v in views):
            return vec.reshape(-1).copy()
        return np.concatenate([a.reshape(-1) for a in out])

    def from_vector(self, vec):
        self._build(MeshLayout(self.mesh), np.asarray(vec, dtype=np.float64))
        return self

    def to_file(self, file_path="projection.npy", write_mesh=True, mesh_file_path="mesh.json"):
        if write_mesh:
            self.mesh.to_file(mesh_file_path)
        self.to_vector().tofile(file_path)

    def __eq__(self, other):
        return self.mesh == other.mesh and self.cols == other.cols


def from_file(mesh_file_path="mesh.json", projection_file_path="projection.npy"):
    """dg/projection/from_file.py:14-21"""
    mesh = _mesh.from_file(mesh_file_path)
    proj = Projection(mesh, None)
    proj.from_vector(np.fromfile(projection_file_path))
    return proj
