"""The Method of Moving Asymptotes with its n-sized work on the device (loadpath/mma.py:31-214).

`MMA(n, m, xmin=0.0, xmax=1.0, move=0.2, c=1000.0, asyinit=0.5, asyincr=1.2, asydecr=0.7)` with
`.update(x, f0, df0, f, df) -> xnew` and `.tighten(factor)`, as loadpath's class: the problem

    minimize    f0(x) + a0 z + sum_i (c_i y_i + 0.5 d_i y_i^2)
    subject to  f_i(x) - a_i z - y_i <= 0,   xmin <= x <= xmax,  y_i >= 0, z >= 0

with a0 = 1, a_i = 0, d_i = 1, solved each iteration by Svanberg's primal-dual interior-point
method on the convex separable approximation built from moving asymptotes. The design, the
asymptotes, the approximation's terms and the subsolver's variables live on the device, and so do its
loops (epsi from 1 down to 1e-7, Newton steps, the line search of up to 50 halvings), in the
reference's order: a graph's while node whose body is two passes over the n-sized variables
(lp_mma.cu), each followed by one block that does the m-sized part and the (m + 1) x (m + 1) Newton
system. The host launches it and reads the outcome once. m <= 8.

x, df0 and df may be numpy arrays (copied to the device; the result comes back as numpy) or
float64 CUDA tensors (the result is a CUDA tensor).
"""
from __future__ import annotations

import ctypes

import numpy as np
import torch

from ._lib import add_launches, launches, lib
from .grid import capturing, free_late, free_later, recording, stream_handle

__all__ = ["MMA"]

MAXM = 8


def _mround(m):
    return 1 if m <= 1 else 2 if m <= 2 else 4 if m <= 4 else 8


class MMA:
    def __init__(self, n, m, xmin=0.0, xmax=1.0, move=0.2, c=1000.0, asyinit=0.5, asyincr=1.2, asydecr=0.7,
                 device="cuda"):
        if not 1 <= m <= MAXM:
            raise ValueError(f"MMA on the device takes 1 <= m <= {MAXM} constraints, got {m}")
        self.n, self.m = int(n), int(m)
        self.M = _mround(self.m)
        self.device = torch.device(device)
        dev = dict(dtype=torch.float64, device=self.device)
        n = self.n

        def vec(v):
            return torch.as_tensor(np.broadcast_to(np.asarray(v, float), (n,)).copy(), **dev)

        self.xmin, self.xmax = vec(xmin), vec(xmax)
        self.move = float(move)
        self.a0 = 1.0
        self.a = np.zeros(m)
        self.c = np.full(m, float(c))
        self.d = np.ones(m)
        self.asyinit, self.asyincr, self.asydecr = float(asyinit), float(asyincr), float(asydecr)
        self.iter = 0
        self.lam = None
        z = lambda *shape: torch.zeros(shape if shape else (n,), **dev)  # noqa: E731
        self._x, self.low, self.upp, self._xold1, self._xold2 = z(), z(), z(), z(), z()
        self._alfa, self._beta, self._p0, self._q0 = z(), z(), z(), z()
        self._P, self._Q, self._df = z(m, n), z(m, n), z(m, n)
        self._df0, self._xnew = z(), z()
        self._sets = [(z(), z(), z()), (z(), z(), z())]   # (x, xsi, eta) of the subsolver, two sets
        self._part = torch.zeros(int(lib().lpb_mma_part_len(m)), **dev)
        self._out = torch.zeros(64, **dev)
        self._state = torch.zeros(int(lib().lpb_mma_state_len()), **dev)
        self._exec = None
        self._have_asy = False
        self._have_old = False

    # -- reference API ------------------------------------------------------------------------
    def tighten(self, factor):
        """Pull the asymptotes toward the last design by `factor` (loadpath/mma.py:48-55)."""
        if self._have_old and self._have_asy:
            self.low.copy_(self._xold1 - factor * (self._xold1 - self.low))
            self.upp.copy_(self._xold1 + factor * (self.upp - self._xold1))

    def update(self, x, f0, df0, f, df):
        """One MMA step (loadpath/mma.py:57-112); returns the new design."""
        L = lib()
        st = stream_handle()
        n, m = self.n, self.m
        host = not isinstance(x, torch.Tensor)
        self._x.copy_(torch.as_tensor(np.asarray(x, float) if host else x).reshape(n))
        self._df0.copy_(torch.as_tensor(np.asarray(df0, float) if not isinstance(df0, torch.Tensor) else df0).reshape(n))
        self._df.copy_(torch.as_tensor(np.asarray(df, float) if not isinstance(df, torch.Tensor) else df).reshape(m, n))
        f = np.nan_to_num(np.asarray(f, float).reshape(m), nan=1e6, posinf=1e6, neginf=-1e6)
        self.iter += 1
        init = self.iter <= 2 or not self._have_asy
        L.lpb_mma_prepare(n, m, self._x.data_ptr(), self.xmin.data_ptr(), self.xmax.data_ptr(), self.low.data_ptr(),
                          self.upp.data_ptr(), None if init else self._xold1.data_ptr(),
                          None if init else self._xold2.data_ptr(), int(init), self.asyinit, self.asyincr,
                          self.asydecr, self.move, self._df0.data_ptr(), self._df.data_ptr(), self._alfa.data_ptr(),
                          self._beta.data_ptr(), self._p0.data_ptr(), self._q0.data_ptr(), self._P.data_ptr(),
                          self._Q.data_ptr(), self._part.data_ptr(), self._out.data_ptr(), st)
        self._have_asy = True
        xs = self._subsolv(f)
        L.lpb_mma_finish(n, xs.data_ptr(), self._x.data_ptr(), self._alfa.data_ptr(), self._beta.data_ptr(),
                         self._xnew.data_ptr(), st)
        self._xold2.copy_(self._xold1 if self._have_old else self._x)
        self._xold1.copy_(self._x)
        self._have_old = True
        return self._xnew.cpu().numpy() if host else self._xnew.clone()

    # -- the subproblem (loadpath/mma.py:114-214) ---------------------------------------------
    def _loop(self):
        """The interior-point loops as a graph with one while node, captured at the first update and again
        when a buffer it names was replaced (a caller may restore low and upp)."""
        bufs = [t.data_ptr() for t in (self.low, self.upp, self._alfa, self._beta, self._p0, self._q0, self._P, self._Q,
                                       *self._sets[0], *self._sets[1], self._state, self._part)]
        if self._exec is None or self._exec_bufs != bufs:
            self._free_loop()
            L = lib()
            c0 = launches()
            with torch.cuda.device(self.device), torch.cuda.stream(torch.cuda.Stream(self.device)), recording():
                st = stream_handle()
                handle, outer, exec_ = ctypes.c_longlong(), ctypes.c_void_p(), ctypes.c_void_p()
                L.lpb_while_begin(st, ctypes.byref(handle), ctypes.byref(outer))
                try:
                    L.lpb_mma_loop_body(handle.value, self.n, self.m, *bufs, st)
                finally:
                    L.lpb_while_end(st, outer, ctypes.byref(exec_))
            self._body = launches() - c0
            add_launches(-self._body)      # recorded, not run
            self._exec, self._exec_bufs = exec_, bufs
        return self._exec

    def _subsolv(self, f, epsimin=1e-7):
        """The subproblem of b = out - f; returns the solution's x."""
        L = lib()
        st = stream_handle()
        x0, xsi0, eta0 = self._sets[0]
        # (d may be one number for all constraints; a and c have a value each)
        host = [np.ascontiguousarray(v, float) for v in (self.a, self.c, np.broadcast_to(self.d, (self.m,)), f)]
        if any(v.shape != (self.m,) for v in host):
            raise ValueError(f"a and c take {self.m} values each")
        L.lpb_mma_sub_init(self.n, self._alfa.data_ptr(), self._beta.data_ptr(), x0.data_ptr(), xsi0.data_ptr(),
                           eta0.data_ptr(), st)
        L.lpb_mma_loop_begin(self.m, self._state.data_ptr(), self._out.data_ptr(), *(v.ctypes.data for v in host),
                             float(self.a0), float(epsimin), st)
        L.lpb_graph_launch(self._loop(), st)
        o = self._state[:16].cpu().numpy()
        add_launches(self._body * int(o[10]))
        if o[8] == 2:
            raise np.linalg.LinAlgError("Singular matrix")
        self.lam = o[:self.m].copy()
        return self._sets[int(o[9])][0]

    def _free_loop(self):
        if self._exec is not None:
            exec_, self._exec = self._exec, None
            torch.cuda.synchronize(self.device)
            lib().lpb_graph_free(exec_)

    def __getstate__(self):
        """Copies and pickles capture a graph of their own."""
        return dict(self.__dict__, _exec=None)

    def __del__(self):
        if getattr(self, "_exec", None) is not None:
            try:
                if capturing():
                    free_later(self.device, lib().lpb_graph_free, [self._exec])
                else:
                    self._free_loop()
                    free_late()
            except Exception:
                pass
