"""Differentiable deltaSPH rollouts of a free fluid (the oscillating drop): forward steps and
their discrete adjoint on the GPU, with checkpointing.

The step is the reference's deltaSPH right-hand side (src/deltaSPH.py:146-200: point
source or gravity, continuity, MOG density diffusion, Tait pressure, artificial and laminar
viscosity) integrated by semi-implicit Euler (src/simulationBase.py:647-652).  Each step
searches neighbors on the GPU (the reference predicate) and advances the state in one launch
(`sph_drop_search`, `sph_drop_step`); the adjoint (`sph_drop_adjoint_step`) runs the steps
backwards, over recorded states or (`vjp`) recomputing each checkpoint segment's states
forward first.  A rollout waits for the device before its first step (the grid) and after its last (the
status).  Scalars are float64 (default) or float32; the search always sees float32 positions,
as the reference's does.  `DropRollout.pairs` and `step` work on the reference's own (i, j)-ordered lists.

Gradients are with respect to the initial velocity field and the artificial viscosity alpha.
`DropRolloutFunction` puts the rollout behind torch.autograd: its forward records every
step's neighbor list and state (a tenth of the list's memory), and its backward runs the
adjoint kernels backwards over them.
"""
from __future__ import annotations

import ctypes

import numpy as np
import torch

from . import _native as N
from .search import MAX_CELLS, GridSearch, _f2, grid_from_words
from .sim import SphParamsC


ROW_SLOTS = 1 << 26   # slots of one step's rows (256 MB) up to which a rollout without a record doubles them


class DropRollout:
    """A drop's rollouts and their gradients from one start.  `checkpoint_every` is the spacing of the states
    that rollout(checkpoints=True) keeps and vjp starts its segments from; loss_and_grad and
    DropRolloutFunction record every step's state instead."""

    def __init__(self, scene: dict, c0: float, dt: float, kinematic: float = 0.001, delta: float = 0.1,
                 rest_density: float = 1000.0, gravity=(0.0, 0.0), point_source: bool = True,
                 point_magnitude: float = 1.0, fp64: bool = True, checkpoint_every: int = 20, device=None,
                 point_center=(0.0, 0.0)):
        self.dev = torch.device(device or torch.device("cuda", torch.cuda.current_device()))
        self.fp64 = bool(fp64)
        self.dtype = torch.float64 if fp64 else torch.float32
        t = lambda a: torch.as_tensor(np.asarray(a), dtype=self.dtype, device=self.dev).contiguous()
        self.n = len(scene["pos"])
        self.x0 = t(scene["pos"]).reshape(self.n, 2)
        self.rho0 = t(scene["rho"])
        self.area = t(scene["area"])
        self.support32 = torch.as_tensor(np.asarray(scene["support"], np.float32), device=self.dev).contiguous()
        self.h = float(np.float32(scene["support"][0]))
        self.vmin = np.asarray(scene["vmin"], np.float32)
        self.vmax = np.asarray(scene["vmax"], np.float32)
        self.dt = float(dt)
        self.every = int(checkpoint_every)
        self.P = SphParamsC()
        P = self.P
        P.support = self.h
        P.rest_density = rest_density
        P.c0 = c0
        P.gamma = 7.0
        P.delta = delta
        P.kinematic = kinematic
        P.gravity[0], P.gravity[1] = gravity
        P.point_source = int(point_source)
        P.point_magnitude = point_magnitude
        P.point_center[0], P.point_center[1] = point_center
        P.density_diffusion = 1            # MOG
        self.search = GridSearch(self.dev)
        self.acc = torch.empty((self.n, 2), dtype=self.dtype, device=self.dev)
        self.dpdt = torch.empty(self.n, dtype=self.dtype, device=self.dev)
        self.steps_run = 0
        # slots of a row: a support's area over a particle's, a quarter more for denser packing
        a = float(np.mean(np.asarray(scene["area"], np.float64)))
        per = np.pi * self.h * self.h / a if a > 0 else 32.0
        self._row_cap = int(min(max(1.25 * per + 8.0, 16.0), 512.0)) + 7 & ~7 if np.isfinite(per) else 32

    # ------------------------------------------------------------------ forward
    def pairs(self, x):
        """(row offsets int32 [n+1], columns int64 [P]) of the reference pair list at x."""
        x32 = x.to(torch.float32).contiguous()
        res = self.search.run(x32, self.support32, kernel_support=self.h, density=False, min_coord=self.vmin,
                              max_coord=self.vmax)
        nb, _, _ = res.to_coo(distances=False)
        rows = nb[0].contiguous()
        cols = nb[1].contiguous()
        off = torch.empty(self.n + 1, dtype=torch.int32, device=self.dev)
        N.call("sph_row_offsets", N.ptr(rows), rows.shape[0], self.n, N.ptr(off), N.stream_ptr())
        return off, cols

    def step(self, x, v, rho, alpha, pairs=None):
        """Advance (x, v, rho) in place by one step; returns the pairs it used."""
        off, cols = pairs or self.pairs(x)
        self.P.alpha = float(alpha)
        st = N.stream_ptr()
        N.call("sph_drop_rhs", int(self.fp64), self.n, N.ptr(off), N.ptr(cols), N.ptr(x), N.ptr(v), N.ptr(rho),
               N.ptr(self.area), ctypes.byref(self.P), N.ptr(self.acc), N.ptr(self.dpdt), st)
        N.call("sph_drop_integrate", int(self.fp64), self.n, N.ptr(x), N.ptr(v), N.ptr(rho), N.ptr(self.acc),
               N.ptr(self.dpdt), self.dt, float(self.P.rest_density), st)
        self.steps_run += 1
        return off, cols

    def _search_plan(self, x32):
        """A rollout's search: the grid (given domain and constant supports, so it holds for every
        step) with the status word behind it, the cell capacity and the scratch."""
        lib, st = N.load(), N.stream_ptr()
        words = torch.zeros(9, dtype=torch.int32, device=self.dev)
        part = torch.empty((lib.sph_grid_scratch_bytes(self.n) + 7) // 8, dtype=torch.int64, device=self.dev)
        N.call("sph_grid_build", N.ptr(x32), N.ptr(self.support32), self.n, _f2(self.vmin), _f2(self.vmax), MAX_CELLS,
               N.ptr(words), N.ptr(words) + 32, N.ptr(part), part.numel() * 8, st)
        *grid, flags = N.read_i32(words)
        if flags:
            raise N.SPHError(f"neighbor search: {N.decode_flags(flags)}")
        cells = max(grid_from_words(grid)["num_cells"], 1)
        size = lib.sph_drop_search_scratch_bytes(self.n, cells)
        return words, cells, torch.zeros((size + 7) // 8, dtype=torch.int64, device=self.dev)

    def _advance(self, state, pr):
        """The state after one step with the pairs pr = (offsets, int32 columns)."""
        out = tuple(torch.empty_like(t) for t in state)
        off, cols = pr
        N.call("sph_drop_step", int(self.fp64), self.n, N.ptr(off), N.ptr(cols), 0, *map(N.ptr, state),
               N.ptr(self.area), ctypes.byref(self.P), self.dt, *map(N.ptr, out), None, N.stream_ptr())
        self.steps_run += 1
        return out

    def _forward(self, v0, alpha, steps, checkpoints=False, record=False):
        """(final state, checkpoints, record of every step), the steps without host waits.

        The rows' slots are sized from the particles' areas with headroom; a step that overflows
        one has the rollout run again: with twice as many where half the rows need them (the slots
        then take at most twice the memory of the reference's int64 lists, usually the same) or
        one step's are a small buffer, else (particles gathered in places, whose rows would cost
        every row of every step their length) over lists of exact length with a host wait per
        step.  A float32 rollout's rows are in increasing order, the order its sums are defined
        in.  A record holds the pairs and the state of every step: the states take a tenth of the
        pairs' memory, and the backward pass neither searches nor steps again."""
        self.P.alpha = float(alpha)
        start = (self.x0.clone(), v0.to(self.dtype).reshape(self.n, 2).clone(memory_format=torch.contiguous_format),
                 self.rho0.clone())
        if steps <= 0:
            return start, {}, None
        n, new = self.n, lambda *shape: torch.empty(shape, dtype=self.dtype, device=self.dev)
        i32 = lambda *shape: torch.empty(shape, dtype=torch.int32, device=self.dev)
        x32 = self.x0.to(torch.float32, copy=True).contiguous()
        words, cells, scratch = self._search_plan(x32)
        status = words[8:]
        st, P, area = N.stream_ptr(), ctypes.byref(self.P), N.ptr(self.area)
        sup, gp, sp, scr, scr_bytes, xp = (N.ptr(self.support32), N.ptr(words), N.ptr(status), N.ptr(scratch),
                                           scratch.numel() * 8, N.ptr(x32))
        slots = steps - 1 if record else min(steps - 1, 2)   # of the states between the first and the last
        while True:
            cap = self._row_cap
            rows = steps if record else 1
            counts, cols = i32(rows, n), i32(rows, n * cap)
            # (rows that one block cannot order by itself are ordered from a second array)
            second = None if self.fp64 or cap <= 512 else i32(n * cap)
            mid, end, ck = (new(slots, n, 2), new(slots, n, 2), new(slots, n)), tuple(map(torch.empty_like, start)), {}
            at = lambda k: [N.ptr(t) for t in start] if k == 0 else [N.ptr(t) for t in end] if k == steps else \
                [t.data_ptr() + (k - 1) % slots * t.stride(0) * t.element_size() for t in mid]
            state = at(0)
            for k in range(steps):
                if checkpoints and k % self.every == 0:
                    ck[k] = tuple(t[(k - 1) % slots].clone() for t in mid) if k else start
                r = k if record else 0
                num, col = counts.data_ptr() + r * n * 4, cols.data_ptr() + r * n * cap * 4
                N.call("sph_drop_search", xp, sup, n, gp, cells, num, cap, col, int(not self.fp64), N.ptr(second), sp, scr,
                       scr_bytes, st)
                after = at(k + 1)
                N.call("sph_drop_step", int(self.fp64), n, num, col, cap, *state, area, P, self.dt, *after, xp, st)
                state = after
            self.steps_run += steps
            flags = int(status.item())
            if not flags & N.SPH_FLAG_PAIR_CAPACITY:
                break
            long_rows = float((counts == 0).sum(1).max()) / n   # (a row that fits holds its particle)
            del counts, cols, second, mid, end, at
            if long_rows < 0.5 and (record or 2 * cap * n > ROW_SLOTS):
                return self._forward_lists(start, steps, checkpoints, record)
            self._row_cap = 2 * cap
            status.zero_()
            x32.copy_(self.x0)
        if flags:
            raise N.SPHError(f"neighbor search: {N.decode_flags(flags)}")
        return end, ck, (start, mid, counts, cols, cap) if record else None

    def _forward_lists(self, state, steps, checkpoints, record):
        """_forward over (i, j)-ordered lists of the rows' exact lengths; the record is a list of
        every step's (state, (offsets, int32 columns))."""
        ck, rec = {}, []
        for k in range(steps):
            if checkpoints and k % self.every == 0:
                ck[k] = state
            off, cols = self.pairs(state[0])
            pr = (off, cols.to(torch.int32))
            if record:
                rec.append((state, pr))
            state = self._advance(state, pr)
        return state, ck, rec if record else None

    def rollout(self, v0, alpha, steps, checkpoints=False, record_pairs=False):
        """Final positions after `steps` steps from (x0, v0, rho0) and the checkpoints (the states
        at every `checkpoint_every`-th step, when asked for); with record_pairs also the list of
        every step's (offsets, columns), in the reference's (i, j) order."""
        if not record_pairs:
            state, ck, _ = self._forward(v0, alpha, steps, checkpoints)
            return state[0], ck
        x = self.x0.clone()
        v = v0.to(self.dtype).reshape(self.n, 2).clone()
        rho = self.rho0.clone()
        ck = {}
        pairs = []
        for k in range(steps):
            if checkpoints and k % self.every == 0:
                ck[k] = (x.clone(), v.clone(), rho.clone())
            pairs.append(self.step(x, v, rho, alpha))
        return x, ck, pairs

    # ------------------------------------------------------------------ adjoint
    def vjp(self, ck, alpha, steps, grad_x, pairs=None):
        """Vector-Jacobian product of the rollout: given d(objective)/d(x_T) = grad_x [n, 2],
        returns (d/d v0 [n, 2], d/d alpha).  Each checkpoint segment's states are recomputed
        forward from its checkpoint, with the recorded pair lists when given (else searched
        again), and the adjoint kernels run the segment's steps backwards."""
        lx = grad_x.to(self.dtype).reshape(self.n, 2).contiguous().clone()
        lv = torch.zeros_like(lx)
        lr = torch.zeros_like(self.rho0)
        nx, nv, nr = torch.empty_like(lx), torch.empty_like(lv), torch.empty_like(lr)
        dalpha = torch.zeros(self.n, dtype=self.dtype, device=self.dev)
        self.P.alpha = float(alpha)
        for s0 in sorted(ck, reverse=True):
            s1 = min(s0 + self.every, steps)
            state = ck[s0]
            seg = []
            for k in range(s0, s1):          # recompute the segment's states
                if pairs is not None:
                    off, cols = pairs[k]
                    pr = (off, cols if cols.dtype == torch.int32 else cols.to(torch.int32))
                else:
                    off, cols = self.pairs(state[0])
                    pr = (off, cols.to(torch.int32))
                seg.append((state, pr))
                if k + 1 < s1:
                    state = self._advance(state, pr)
            for (xs, vs, rs), (off, cols) in reversed(seg):
                N.call("sph_drop_adjoint_step", int(self.fp64), self.n, N.ptr(off), N.ptr(cols), 0,
                       N.ptr(xs), N.ptr(vs), N.ptr(rs), N.ptr(self.area), ctypes.byref(self.P), self.dt, N.ptr(lx),
                       N.ptr(lv), N.ptr(lr), N.ptr(nx), N.ptr(nv), N.ptr(nr), N.ptr(dalpha), N.stream_ptr())
                lx, nx = nx, lx
                lv, nv = nv, lv
                lr, nr = nr, lr
        return lv, dalpha.sum()

    def _backward(self, record, alpha, steps, grad_x):
        """vjp over a forward pass's record."""
        lx = grad_x.to(self.dtype).reshape(self.n, 2).contiguous().clone()
        cur = (lx, torch.zeros_like(lx), torch.zeros_like(self.rho0))
        nxt = tuple(map(torch.empty_like, cur))
        dalpha = torch.zeros(self.n, dtype=self.dtype, device=self.dev)
        self.P.alpha = float(alpha)
        st, P, area, da = N.stream_ptr(), ctypes.byref(self.P), N.ptr(self.area), N.ptr(dalpha)
        a, b = [N.ptr(t) for t in cur], [N.ptr(t) for t in nxt]
        for k in reversed(range(steps)):
            if isinstance(record, list):
                state, pr = record[k]
                pairs, state = (*map(N.ptr, pr), 0), map(N.ptr, state)
            else:
                start, mid, counts, cols, cap = record
                pairs = (counts.data_ptr() + k * self.n * 4, cols.data_ptr() + k * self.n * cap * 4, cap)
                state = [t.data_ptr() + (k - 1) * t.stride(0) * t.element_size() for t in mid] if k else map(N.ptr, start)
            N.call("sph_drop_adjoint_step", int(self.fp64), self.n, *pairs, *state, area, P, self.dt, *a, *b, da, st)
            a, b = b, a
            cur, nxt = nxt, cur
        return cur[1], dalpha.sum()

    def loss_and_grad(self, v0, alpha, target, steps):
        """Loss mean_i |x_T,i - target_i|^2 and its gradients with respect to v0 [n, 2] and alpha."""
        (xT, *_), _, record = self._forward(v0, alpha, steps, record=True)
        diff = xT - target.to(self.dtype)
        loss = float((diff * diff).sum().item()) / self.n
        lv, da = self._backward(record, alpha, steps, (2.0 / self.n) * diff)
        return loss, lv, float(da.item())

    def loss(self, v0, alpha, target, steps):
        xT, _ = self.rollout(v0, alpha, steps)
        d = xT - target.to(self.dtype)
        return float((d * d).sum().item()) / self.n


class DropRolloutFunction(torch.autograd.Function):
    """Final positions x_T [n, 2] of a `steps`-step DropRollout as a differentiable function of
    the initial velocities v0 [n, 2] and the artificial viscosity alpha (0-d tensor).

    Forward: the GPU rollout, recording each step's neighbor list and state.  Backward: the
    adjoint of each step over the record (sph_drop_adjoint_step).  The rollout's precision (float32 or float64) is the
    rollout's; gradients come back in the inputs' dtypes."""

    @staticmethod
    def forward(ctx, v0, alpha, rollout, steps):
        a = float(alpha)
        (xT, *_), _, ctx.record = rollout._forward(v0.detach(), a, int(steps), record=True)
        ctx.rollout, ctx.alpha, ctx.steps = rollout, a, int(steps)
        ctx.v_dtype, ctx.a_dtype = v0.dtype, (alpha.dtype if isinstance(alpha, torch.Tensor) else torch.float64)
        ctx.a_device = alpha.device if isinstance(alpha, torch.Tensor) else v0.device
        return xT

    @staticmethod
    def backward(ctx, grad_x):
        gv, ga = ctx.rollout._backward(ctx.record, ctx.alpha, ctx.steps, grad_x)
        gv = gv.to(ctx.v_dtype) if ctx.needs_input_grad[0] else None
        ga = ga.to(device=ctx.a_device, dtype=ctx.a_dtype) if ctx.needs_input_grad[1] else None
        return gv, ga, None, None


def drop_rollout(rollout: DropRollout, v0: torch.Tensor, alpha, steps: int) -> torch.Tensor:
    """x_T = DropRolloutFunction.apply(v0, alpha, rollout, steps)."""
    if not isinstance(alpha, torch.Tensor):
        alpha = torch.tensor(float(alpha), dtype=torch.float64, device=v0.device)
    return DropRolloutFunction.apply(v0, alpha, rollout, steps)
