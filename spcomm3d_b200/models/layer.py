"""Pipelines built from the two distributed kernels.

`SddmmSpmmStep`  one SDDMM followed by one SpMM on the same sparse matrix with
                 its stored values: the unit the benchmarks time (the
                 reference runs the two kernels as separate programs,
                 miniapp/bench_both.cpp and miniapp/bench_spmm.cpp, or back to
                 back in miniapp/main_combined.cpp:165-281).
`GatLayer`       attention-style chain: edge scores C = S o (A B^T), then
                 Y = C X with the scores as the sparse values.  The scores are
                 summed along the Z fiber and then shared by the whole fiber,
                 because every Z layer multiplies the full block with its own
                 slice of X's columns.
"""
from __future__ import annotations

import numpy as np
import torch
import torch.distributed as dist

from ..parallel.mesh import split_nnz
from .dist_ops import DistSDDMM, DistSpMM

STREAM_A, STREAM_B = 1, 2


def _bind_pair(old, sddmm, spmm):
    """Two bound calls as one, in place of `old`."""
    from ..ops.cuda_ops import BoundPair
    if old is not None:
        old.retire()
    return BoundPair(sddmm, spmm)


class SddmmSpmmStep:
    _pair = None   # the two bound calls as one

    def __init__(self, plan, groups, k, dtype=torch.float32, device="cuda", variant="sparseNRB", seed=0,
                 **kw):
        self.plan, self.k, self.seed = plan, k, seed
        self.device = torch.device(device)
        self.sddmm = DistSDDMM(plan, groups, k, dtype, device, variant, **kw)
        self.spmm = DistSpMM(plan, groups, k, dtype, device, variant, **kw)
        self.host = None
        self._native_step = None
        if self.sddmm._single and self.spmm._single:
            self._bind()

    def __getstate__(self):
        return {**self.__dict__, "_native_step": None, "_pair": None}   # bound to this step's tensors, like the operators' calls

    def fill_device_operands(self):
        """A, B (and X = B) generated on the device from the seed."""
        sd, sp, p = self.sddmm, self.spmm, self.plan
        if self.device.type == "cuda":
            from ..ops import cuda_ops
            ga = torch.from_numpy(p.row.owned_gids).to(self.device)
            gb = torch.from_numpy(p.col.owned_gids).to(self.device)
            cuda_ops.fill_rows(ga, self.k, sd.k_off, sd.A_owned, seed=self.seed, stream=STREAM_A)
            cuda_ops.fill_rows(gb, self.k, sd.k_off, sd.B_owned, seed=self.seed, stream=STREAM_B)
            sp.X_owned.copy_(sd.B_owned)
        else:
            sd.fill_owned(sd.A_owned, p.row.owned_gids, seed=self.seed, stream=STREAM_A)
            sd.fill_owned(sd.B_owned, p.col.owned_gids, seed=self.seed, stream=STREAM_B)
            sp.X_owned.copy_(sd.B_owned)

    def _bind(self):
        self._pair = _bind_pair(self._pair, self.sddmm._bind(), self.spmm._bind())
        self._pair.c = self.sddmm._slice
        return self._pair

    def run_device(self):
        sd, sp, pair = self.sddmm, self.spmm, self._pair
        if sd._single and sp._single:
            if pair is None or not pair.bound_to(sd.rowidx, sd.colidx, sd.vals, sd.A_loc, sd.B_loc, sd.partial,
                                                 sp.rowptr, sp.colidx, sp.vals, sp.X_loc, sp.Y_loc):
                pair = self._bind()
            pair.launch()
            return pair.c, sp.Y_owned
        return sd.run_async(), sp.run_async()

    # ---- end to end: operands start in pinned host memory -----------------
    def make_host_operands(self):
        sd = self.sddmm
        self._dev_made = {"A": sd.A_owned, "B": sd.B_owned}
        # padded rows (fused variant) travel with their padding: one contiguous copy each
        full = {n: self._whole_rows(t).cpu() for n, t in self._dev_made.items()}
        if self.device.type == "cuda":
            full = {n: t.pin_memory() for n, t in full.items()}
        self.host = {n: t[:, :sd.k_loc] for n, t in full.items()}
        self._host_made = dict(self.host)
        self._native_step = None
        self._sums = torch.zeros(2, dtype=torch.float64, device=self.device)
        self._bound_step()   # the pinned buffer, the stream and the events of the one-call form are made here
        return self.host

    @staticmethod
    def _whole_rows(t):
        """The rows of `t` with what lies between one and the next."""
        return t.as_strided((t.shape[0], t.stride(0)), (t.stride(0), 1)) if t.shape[0] > 1 else t

    def _upload(self, name, dst):
        src = self.host[name]
        if src is self._host_made[name] and dst is self._dev_made[name]:
            src, dst = self._whole_rows(src), self._whole_rows(dst)
        dst.copy_(src, non_blocking=True)

    @property
    def h2d_bytes(self):
        made = [t if t is not self._host_made[n] else self._whole_rows(t) for n, t in self.host.items()]
        return int(sum(t.numel() * t.element_size() for t in made))

    @property
    def d2h_bytes(self):
        return 16

    def _bound_step(self):
        """The step of a single GPU as one native call (bound again when an operator had a tensor replaced), or None
        where that call would not be this step: several ranks, operands of the user's own on the host, or operands on
        the device that are not those that the copies go to."""
        sd, sp, h = self.sddmm, self.spmm, self.host
        if not (sd._single and sp._single) or any(h[n] is not t for n, t in self._host_made.items()):
            return None
        for loc, owned, like in ((sd.A_loc, sd.A_owned, h["A"]), (sd.B_loc, sd.B_owned, h["B"]),
                                 (sp.X_loc, sp.X_owned, h["B"]), (sp.Y_loc, sp.Y_owned, sp.Y_owned)):
            if (loc.data_ptr() != owned.data_ptr() or not loc.shape == owned.shape == like.shape
                    or loc.dtype != like.dtype or not (loc.is_contiguous() and owned.is_contiguous())):
                return None
        from ..ops import cuda_ops
        bs, bp = sd._bind(), sp._bind()
        if self._native_step is None or self._native_step[0] is not bs or self._native_step[1] is not bp:
            self._native_step = (bs, bp, cuda_ops.HostStep(bs, bp, h["A"], h["B"], sd.A_loc, sd.B_loc, sp.X_loc, sp.Y_loc,
                                                           self.plan.rowptr, self.device))
        return self._native_step[2]

    def run_e2e(self):
        """Copies the step's inputs A and B from pinned host memory (X of the
        SpMM is B: one device-to-device copy), runs SDDMM and SpMM (the SpMM
        overlaps the copy of A) and reads back the checksums of this rank's
        results (two fp64 scalars)."""
        sd, sp = self.sddmm, self.spmm
        native_step = self._bound_step()
        if native_step is not None:
            return native_step.run()
        if self.device.type == "cuda":
            # B first; while A follows on a copy stream the SpMM (which needs only X = B) already runs
            main = torch.cuda.current_stream(self.device)
            if getattr(self, "_copy_stream", None) is None:
                self._copy_stream = torch.cuda.Stream(self.device)
                self._ev_b, self._ev_a = torch.cuda.Event(), torch.cuda.Event()
            self._upload("B", sd.B_owned)
            self._ev_b.record(main)
            self._copy_stream.wait_event(self._ev_b)   # also orders this copy of A after the previous step's SDDMM
            with torch.cuda.stream(self._copy_stream):
                self._upload("A", sd.A_owned)
                self._ev_a.record(self._copy_stream)
            sp.X_owned.copy_(sd.B_owned)
            y = sp.run_async()
            main.wait_event(self._ev_a)
            c = sd.run_async()
        else:
            self._upload("A", sd.A_owned)
            self._upload("B", sd.B_owned)
            sp.X_owned.copy_(sd.B_owned)
            c = sd.run_async()
            y = sp.run_async()
        if self.device.type == "cuda":
            from ..ops import cuda_ops
            self._sums[0:1].copy_(cuda_ops.checksum(c))
            self._sums[1:2].copy_(cuda_ops.checksum(y.reshape(-1)))
        else:
            self._sums[0], self._sums[1] = c.double().sum(), y.double().sum()
        return self._sums.cpu().tolist()

    # ---- health, timing breakdown, shutdown --------------------------------
    def check(self):
        """Synchronises and raises `FusedStatusError` if a fused kernel of either op recorded a bad index
        or a wait that ran out since the last check (the asynchronous run path does not look)."""
        for op in (self.sddmm, self.spmm):
            f = getattr(op, "_fused", None)
            if f is not None:
                f.check()

    def phase_ms(self):
        """In-kernel time stamps of the last fused launches: {"sddmm": {"pull", "main", "total"}, "spmm": ...}
        in milliseconds, or None for the library variants."""
        if getattr(self.sddmm, "_fused", None) is None:
            return None
        return {"sddmm": self.sddmm._fused.phase_ms(), "spmm": self.spmm._fused.phase_ms()}

    def local_kernel_ms(self, iters: int = 5):
        """(sddmm_ms, spmm_ms) of the plain local kernels on this rank's block with every dense row already
        in local memory: what the distributed ops would cost if communication were free."""
        from ..ops import local
        sd, sp, p = self.sddmm, self.spmm, self.plan
        dev, dt, kl = self.device, sd.dtype, sd.k_loc
        f = getattr(sd, "_fused", None)
        A = f._A_full[:, :kl] if f is not None else sd.A_loc
        Y = torch.empty(p.row.n_local, kl, dtype=dt, device=dev)
        sched = sp.sched
        if sched is None and dev.type == "cuda":
            sched = sp._fused.sched if getattr(sp, "_fused", None) is not None else None
        out = []
        for fn in (lambda: local.sddmm(sd.rowidx, sd.colidx, sd.vals, A, sd.B_loc, out=sd.partial),
                   lambda: local.spmm(sp.rowptr, sp.rowidx, sp.colidx, sp.vals, sp.X_loc, Y, 0.0, sched)):
            fn()
            if dev.type == "cuda":
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                for _ in range(iters):
                    fn()
                b.record()
                torch.cuda.synchronize(dev)
                out.append(a.elapsed_time(b) / iters)
            else:
                import time
                t0 = time.perf_counter()
                for _ in range(iters):
                    fn()
                out.append((time.perf_counter() - t0) * 1e3 / iters)
        return tuple(out)

    def close(self):
        """Collective shutdown of both ops (see `_Dist3DOp.close`)."""
        self.sddmm.close()
        self.spmm.close()

    def comm_volume_bytes(self):
        """[sddmm expand, sddmm z-reduce, spmm expand, spmm reduce] bytes this
        rank receives per step according to the plan."""
        es = self.sddmm.A_loc.element_size()
        pre, post = (self.sddmm.comm_stats()[p] for p in ("PRE", "POST"))
        z = self.plan.mesh.Z
        zred = (self.plan.nnz - post[1][1]) if z > 1 else 0  # values leaving this rank
        spre, spost = (self.spmm.comm_stats()[p] for p in ("PRE", "POST"))
        return [pre[1][1] * es, zred * es, spre[1][1] * es, spost[1][1] * es]


class GatLayer:
    """Y = (S o (A B^T)) X on the mesh; returns owned rows of Y."""

    _pair = None   # the two bound calls as one

    def __init__(self, plan, groups, k, dtype=torch.float32, device="cpu", variant="sparseNRB", **kw):
        self.plan, self.groups = plan, groups
        self.sddmm = DistSDDMM(plan, groups, k, dtype, device, variant, **kw)
        # the SpMM values change every run (they are the SDDMM scores): no precomputed value panels here
        self.spmm = DistSpMM(plan, groups, k, dtype, device, variant,
                             **{k_: v for k_, v in kw.items() if k_ != "panels"})
        Z = plan.mesh.Z
        self.slices = [split_nnz(plan.nnz, Z, z) for z in range(Z)]
        self.width = self.slices[0][1]
        dev = torch.device(device)
        self._mine = torch.zeros(self.width, dtype=dtype, device=dev)
        self._all = torch.zeros(Z, self.width, dtype=dtype, device=dev)
        self._scores = None
        if self._direct():
            scores = self._bind_scores()
            if self.spmm._single:
                self._pair = _bind_pair(None, scores, self.spmm._bind())
            self.sddmm._bound = None   # (its own call is bound when it runs alone: the scratch is not needed twice)
        # the SpMM wants its values in CSR order; a fused SDDMM stores them in its own order
        order = self.sddmm.value_order
        self._pos = None if order is None else torch.from_numpy(np.ascontiguousarray(order)).to(dev)

    def __getstate__(self):
        return {**self.__dict__, "_scores": None, "_pair": None}   # bound to this layer's tensors, like the operators' calls

    def _direct(self):
        """Whether the kernel of the SDDMM itself can put the scores where the SpMM reads its values, next to the result
        of the SDDMM (which stays what it is when the SpMM's values change)."""
        c, v = self.sddmm.partial, self.spmm.vals
        return (self.sddmm._single and v is not c and v.dtype == c.dtype and v.shape == c.shape and v.is_contiguous()
                and v.device == c.device)

    def _bind_scores(self):
        self._scores = self.sddmm._bind(self._scores, (self.spmm.vals,))
        return self._scores

    def run(self):
        sd, sp = self.sddmm, self.spmm
        if not sd.timer.enabled and sd._single:
            pair = self._pair if sp._single and not sp.timer.enabled else None
            if pair is not None and pair.bound_to(sd.rowidx, sd.colidx, sd.vals, sd.A_loc, sd.B_loc, sd.partial, sp.vals,
                                                  sp.rowptr, sp.colidx, sp.vals, sp.X_loc, sp.Y_loc):
                pair.launch()
                return sp.Y_owned
            if self._direct():
                scores = self._bind_scores()
                if sp._single and not sp.timer.enabled:
                    self._pair = _bind_pair(self._pair, scores, sp._bind())
                    self._pair.launch()
                    return sp.Y_owned
                scores.launch()
                return sp.run()
        c = sd.run()
        Z = self.plan.mesh.Z
        if Z == 1:
            if self._pos is None:
                self.spmm.vals.copy_(c)
            else:
                self.spmm.vals.index_copy_(0, self._pos, c)
        else:
            self._mine[:c.shape[0]].copy_(c)
            dist.all_gather_into_tensor(self._all.view(-1), self._mine, group=self.groups.fiber)
            for z, (o, l) in enumerate(self.slices):
                if self._pos is None:
                    self.spmm.vals[o:o + l].copy_(self._all[z, :l])
                else:
                    self.spmm.vals.index_copy_(0, self._pos[o:o + l], self._all[z, :l])
        self.spmm.values_changed()
        return self.spmm.run()
