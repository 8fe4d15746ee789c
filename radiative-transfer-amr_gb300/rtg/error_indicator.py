"""Error indicators and hp steering of the AMR loop on the GPU.

Mirrors the reference's ``Error_Indicator`` (src/amr/Error_Indicator/
class_Error_Indicator.py:12-28): ``ErrorIndicator(proj, ref_kind, ref_form,
ref_tol)`` with ``error_angular_jump()`` (error/error_angular_jump.py:14-137),
``error_spatial_jump()`` (error/error_spatial_jump.py:17-289),
``col_hp_steer(col_key)`` (col_hp_steer.py:14-64) and
``cell_hp_steer(col_key, cell_key)`` (cell_hp_steer.py:15-48).  After an
``error_*`` call: ``cols[col_key]`` is an ``ErrorIndicatorColumn`` (``error``,
``cells``, ``ref_form``, ``do_ref``) whose ``cells[cell_key]`` are
``ErrorIndicatorCell`` objects, and ``col_max_error``, ``cell_max_error``,
``error`` and ``error_to_resolve`` are set, as in the reference.  The jumps and
the hp estimates run in librtg's kernels (rtg_error_angular_jump,
rtg_error_spatial_jump, rtg_hp_steer); the flags are set on the host in the
reference's loop order.
"""
import ctypes as C
import math

import numpy as np

from . import _lib

INF = float(np.finfo(np.float64).max)   # the reference's consts.INF


class ErrorIndicatorCell:
    def __init__(self, error, ref_form="", do_ref=False):
        self.error = error
        self.ref_form = ref_form
        self.do_ref = do_ref


class ErrorIndicatorColumn:
    def __init__(self, error, cells, ref_form="", do_ref=False):
        self.error = error
        self.cells = cells
        self.ref_form = ref_form
        self.do_ref = do_ref


def _unit_coefficients():
    return (lambda x, y: 1. + 0. * x, lambda x, y: 0. * x, lambda th, ph: 0. * th + 1. / (2. * math.pi))


class ErrorIndicator:
    """``proj``: an ``rtg.Projection`` (or any object with ``mesh`` and
    ``to_vector()``).  ``ctx``: a DeviceContext on the same mesh to reuse
    (for example the one the solve ran on); one with unit coefficients is
    made otherwise (the indicators use only the mesh)."""

    def __init__(self, proj, ref_kind="all", ref_form="hp", ref_tol=(INF, INF), ctx=None):
        from .problem import DeviceContext
        self.proj = proj
        self.ref_kind = ref_kind
        self.ref_form = ref_form
        [self.ang_ref_tol, self.spt_ref_tol] = ref_tol
        self._own = ctx is None
        self.ctx = ctx if ctx is not None else DeviceContext(proj.mesh, *_unit_coefficients())
        self._u = None
        self._lp = None
        self.cols = {}
        self.col_max_error = -INF
        self.cell_max_error = -INF
        self.error = 0.
        self.error_to_resolve = 0.

    # ------------------------------------------------------------- device
    def _u_dev(self):
        if self._u is None:
            self._u = self.ctx.to_device(np.asarray(self.proj.to_vector(), dtype=np.float64))
        return self._u

    def _keys(self):
        lay = self.ctx.layout
        return lay.col_keys, lay.elem_keys

    def _hp(self):
        if self._lp is None:
            torch = self.ctx.torch
            lay = self.ctx.layout
            col_lp = torch.empty(lay.ncols, dtype=torch.float64, device=self.ctx.device)
            cell_lp = torch.empty(lay.nelem, dtype=torch.float64, device=self.ctx.device)
            _lib.check(self.ctx.lib.rtg_hp_steer(self.ctx.h, C.c_void_p(self._u_dev().data_ptr()),
                                                 C.c_void_p(col_lp.data_ptr()), C.c_void_p(cell_lp.data_ptr()),
                                                 None))
            col_keys, elem_keys = self._keys()
            self._lp = (dict(zip(col_keys, col_lp.tolist())), dict(zip(elem_keys, cell_lp.tolist())))
        return self._lp

    # ---------------------------------------------------------- hp steering
    def col_hp_steer(self, col_key):
        """'p' when lp - 1/2 >= (nx + ny)/2, else 'h' (col_hp_steer.py:56-64)."""
        lp = self._hp()[0][col_key]
        nx, ny = self.proj.mesh.cols[col_key].ndofs[:2]
        return "p" if lp - 0.5 >= 0.5 * (nx + ny) else "h"

    def cell_hp_steer(self, col_key, cell_key):
        """'p' when lp - 1/2 >= nth, else 'h' (cell_hp_steer.py:40-48)."""
        lp = self._hp()[1][(col_key, cell_key)]
        nth = self.proj.mesh.cols[col_key].cells[cell_key].ndofs[0]
        return "p" if lp - 0.5 >= float(nth) else "h"

    # ----------------------------------------------------------- indicators
    def error_angular_jump(self):
        torch = self.ctx.torch
        lay = self.ctx.layout
        ce = torch.empty(lay.nelem, dtype=torch.float64, device=self.ctx.device)
        _lib.check(self.ctx.lib.rtg_error_angular_jump(self.ctx.h, C.c_void_p(self._u_dev().data_ptr()),
                                                       C.c_void_p(ce.data_ptr()), None, None))
        ce = ce.tolist()
        err = list(map(math.sqrt, ce))
        col_keys, elem_keys = self._keys()
        start = lay.col_elem_start.tolist()
        cols, col_err, mesh_err = {}, [], 0.
        for i, ck in enumerate(col_keys):
            e0, e1 = start[i], start[i + 1]
            s = 0.
            for v in ce[e0:e1]:
                s += v
                mesh_err += v
            col_err.append(math.sqrt(s))
            cols[ck] = ErrorIndicatorColumn(col_err[i], {elem_keys[e][1]: ErrorIndicatorCell(err[e])
                                                         for e in range(e0, e1)})
        self._finish(cols, col_err, err, mesh_err)

    def error_spatial_jump(self):
        torch = self.ctx.torch
        lay = self.ctx.layout
        cc = torch.empty(lay.ncols, dtype=torch.float64, device=self.ctx.device)
        _lib.check(self.ctx.lib.rtg_error_spatial_jump(self.ctx.h, C.c_void_p(self._u_dev().data_ptr()),
                                                       C.c_void_p(cc.data_ptr()), None))
        cc = cc.tolist()
        col_err = list(map(math.sqrt, cc))
        col_keys, elem_keys = self._keys()
        start = lay.col_elem_start.tolist()
        cols, mesh_err = {}, 0.
        for i, ck in enumerate(col_keys):
            mesh_err += cc[i]
            cols[ck] = ErrorIndicatorColumn(col_err[i], {elem_keys[e][1]: ErrorIndicatorCell(-INF)
                                                         for e in range(start[i], start[i + 1])})
        self._finish(cols, col_err, [-INF] * lay.nelem, mesh_err)

    def _finish(self, cols, col_err, cell_err, mesh_err):
        """Maxima, mesh error and the refinement flags in the reference's
        loop order (error_angular_jump.py:84-137).  Columns and cells are new, their
        do_ref False: only those over a threshold are visited."""
        self.cols = cols
        self.col_max_error = max([-INF, *col_err])
        self.cell_max_error = max([-INF, *cell_err])
        self.error = math.sqrt(mesh_err)
        self.error_to_resolve = 0.
        ang_thr = self.ang_ref_tol * self.cell_max_error
        spt_thr = self.spt_ref_tol * self.col_max_error
        lay = self.ctx.layout
        col_keys, elem_keys = self._keys()
        hits = []      # (column index, -1 or element index): a column, then its cells
        if self.ref_kind in ("spt", "all"):
            hits += [(i, -1) for i, v in enumerate(col_err) if v >= spt_thr]
        if self.ref_kind in ("ang", "all"):
            hits += [(int(lay.elem_col[e]), e) for e, v in enumerate(cell_err) if v >= ang_thr]
        for i, e in sorted(hits):
            ck = col_keys[i]
            if e < 0:
                it, steer = cols[ck], lambda: self.col_hp_steer(ck)
            else:
                kk = elem_keys[e][1]
                it, steer = cols[ck].cells[kk], lambda: self.cell_hp_steer(ck, kk)
            it.do_ref = True
            self.error_to_resolve += it.error
            it.ref_form = steer() if self.ref_form == "hp" else self.ref_form

    def close(self):
        if self._own and self.ctx is not None:
            self.ctx.close()
        self.ctx = None
