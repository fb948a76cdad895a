"""
Learned surrogate for the polydisperse cylinder: log I(q | R, L, R_pd, L_pd,
contrast, q, orientation flag), with the plain kernels as its data source,
its judge and its fallback.

* The network (``csrc/mlp.cu``) is 7 inputs (padded to 16) -> 4 x 256 SiLU
  -> 1, BF16 weights and activations, FP32 accumulation on the tcgen05
  tensor cores, trained here with the project's own forward, backward,
  weight-gradient and Adam kernels.
* Training data: parameter sets drawn uniformly / log-uniformly over the
  domain below, evaluated by the plain engines: flag 1 = the 1D orientation
  average (``cylinder`` Fq, batched engine), flag 0 = the oriented 2D kernel
  at theta = 90, phi = 0 without jitter, with q along qx.
* The intensity is exactly quadratic in the contrast, so the network learns
  y = log I at unit contrast and ``2 log|contrast|`` is added back.
* Predicted error: a second network of the same shape (the error gate,
  same kernels) trained on fresh sets to predict the local envelope of the
  first network's |log I error|, with per-tolerance thresholds calibrated
  on held-out sets judged by the plain FP64 kernel (at most 0.05 % of the
  accepted calibration points off by more than the tolerance).  Points
  whose predicted error exceeds the tolerance (default 1 % in log I), or
  that fall outside the training domain, are recomputed by the plain
  kernel.

Domain: R in [10, 300] A, L in [20, 3000] A, R_pd and L_pd in [0, 0.3]
(gaussian, 35 points, 3 sigma when > 0), contrast in [-5, 5], q in
[1e-3, 0.5] 1/A.
"""

import ctypes as ct
import math
import os

import numpy as np

from ._abi import LIB_DIR

HID = 256
NIN = 16
TM = 128
DOMAIN = dict(radius=(10.0, 300.0), length=(20.0, 3000.0), rpd=(0.0, 0.3),
              lpd=(0.0, 0.3), contrast=(-5.0, 5.0), q=(1e-3, 0.5))
PD_N = 35
#: linear learning-rate warm-up of the training schedule, in steps
WARMUP_STEPS = 200


_LIB = None


def _lib():
    global _LIB
    if _LIB is None:
        _LIB = _load()
    return _LIB


def _load():
    path = os.path.join(LIB_DIR, "libsasb200_mlp.so")
    if not os.path.exists(path):
        raise RuntimeError("surrogate library not built: %s" % path)
    lib = ct.CDLL(path)
    P, I, F = ct.c_void_p, ct.c_int32, ct.c_float
    lib.sasb200_mlp_forward.argtypes = [I, I, P, P, P, P, P, P, P, P, P, P, P]
    lib.sasb200_mlp_backward.argtypes = [I, I, P, P, P, P, P, P, P]
    lib.sasb200_loss_grad.argtypes = [I, I, P, P, F, P, P, P]
    lib.sasb200_adam.argtypes = [I, I, P, P, P, P, F, F, F, F, I, P, P, I, I, P]
    lib.sasb200_lr_schedule.argtypes = [P, P, I, I, F, F, F, P]
    lib.sasb200_col_sums.argtypes = [I, I, P, P, P, P, P]
    lib.sasb200_col_sum_parts.argtypes = [I]
    lib.sasb200_mlp_features.argtypes = [I, I, P, P, P, P, P, P, P, P, P, P]
    lib.sasb200_mlp_pack.argtypes = [P, P, P, P, P, P]
    lib.sasb200_mlp_infer.argtypes = [I, I, P, P, P, P, P, P, P, P, P, P, I, P]
    lib.sasb200_mlp_serve.argtypes = [I, I, P, P, P, P, P, P, P, P, P, P, I, P]
    lib.sasb200_mlp_pack_t.argtypes = [P, P, P, P, P]
    lib.sasb200_mlp_backward_p.argtypes = [I, I, P, P, P, P, P, P, I, P]
    lib.sasb200_mlp_train_pass.argtypes = [P, P]
    lib.sasb200_adam_pack.argtypes = [P]*10 + [F, I, F, F, F, P]
    D = ct.c_double
    lib.sasb200_features_runs.argtypes = [I, I, I] + [P]*6
    lib.sasb200_finish_runs.argtypes = [I, I] + [P]*5 + [D]*7 + [P]*3
    for name in ("sasb200_features_runs", "sasb200_finish_runs",
                 "sasb200_adam_pack",
                 "sasb200_mlp_train_pass",
                 "sasb200_mlp_forward", "sasb200_mlp_backward", "sasb200_loss_grad",
                 "sasb200_adam", "sasb200_mlp_features", "sasb200_mlp_pack",
                 "sasb200_mlp_infer", "sasb200_mlp_serve", "sasb200_mlp_image_bytes",
                 "sasb200_mlp_pack_t", "sasb200_mlp_image_t_bytes", "sasb200_mlp_backward_p",
                 "sasb200_lr_schedule", "sasb200_col_sums", "sasb200_col_sum_parts"):
        getattr(lib, name).restype = I
    lib.sasb200_mlp_last_error.restype = ct.c_char_p
    return lib


#: code of a captured step whose batch names a row that the data set lacks
ROW_OUTSIDE = 5
OUTSIDE = "a row index outside the training data"


def pad128(n):
    return ((n + TM - 1)//TM)*TM


class _Batch(ct.Structure):
    """The batch of a captured training step (sasb200_mlp_batch)."""

    _fields_ = [("idx", ct.c_void_p), ("rows", ct.c_int64), ("x_all", ct.c_void_p),
                ("x_lo_all", ct.c_void_p), ("y_all", ct.c_void_p), ("counters", ct.c_void_p),
                ("sched", ct.c_void_p), ("refused", ct.c_void_p), ("total", ct.c_int32), ("warmup", ct.c_int32),
                ("lr0", ct.c_float), ("b1", ct.c_float), ("b2", ct.c_float)]


class _Pass(ct.Structure):
    """The operands of a gradient pass (sasb200_mlp_pass)."""

    _fields_ = ([(k, ct.c_int32) for k in ("n", "n_pad", "splits")] + [("delta", ct.c_float)]
                + [(k, ct.c_void_p) for k in ("x", "x_lo", "y", "img", "img_t")]
                + [("b", ct.c_void_p*4)]
                + [(k, ct.c_void_p) for k in ("w_out", "b_out", "out", "dout", "row_sums", "z",
                                              "h", "dz")]
                + [("dw", ct.c_void_p*4)]
                + [(k, ct.c_void_p) for k in ("db", "dw_out", "loss", "db_out", "batch", "err")]
                + [("sums", ct.c_int32), ("sum_sizes", ct.c_int32*16),
                   ("sum_splits", ct.c_int32*16), ("sum_parts", ct.c_void_p*16),
                   ("sum_outs", ct.c_void_p*16)])


class MLP:
    """Weights, optimiser state and the device kernels of the surrogate."""

    def __init__(self, device=None, seed=0, stream=None):
        import torch
        self.torch = torch
        self.device = torch.device(device if device is not None else "cuda")
        if self.device.index is None:
            self.device = torch.device("cuda", torch.cuda.current_device())
        self.lib = _lib()
        self.stream = stream if stream is not None else torch.cuda.Stream(self.device)
        rng = np.random.default_rng(seed)
        shapes = [(HID, NIN), (HID, HID), (HID, HID), (HID, HID)]
        f32 = dict(dtype=torch.float32, device=self.device)
        self.W, self.b = [], []
        for l, (o, i) in enumerate(shapes):
            fan_in = 15 if l == 0 else i
            bound = math.sqrt(6.0/fan_in)
            w = rng.uniform(-bound, bound, (o, i))
            if l == 0:
                w[:, 15:] = 0.0
            self.W.append(torch.as_tensor(w, **f32))
            self.b.append(torch.zeros(o, **f32))
        self.w_out = torch.as_tensor(rng.uniform(-1, 1, HID)/math.sqrt(HID), **f32)
        self.b_out = torch.zeros(1, **f32)
        self.params = self.W + self.b + [self.w_out, self.b_out]
        self._sizes = [p.numel() for p in self.params]
        self.m = [torch.zeros_like(p) for p in self.params]
        self.v = [torch.zeros_like(p) for p in self.params]
        self.step_count = 0
        #: partial sums of each weight gradient (see mlp_weight_grads: 14 blocks
        #: per split, one wave of blocks)
        self.splits = 10
        #: Huber threshold of the training loss (<= 0: squared error)
        self.huber = 0.0
        self.err = torch.zeros(1, dtype=torch.int32, device=self.device)
        self.img = torch.empty(self.lib.sasb200_mlp_image_bytes(), dtype=torch.uint8,
                               device=self.device)
        self.img_t = torch.empty(self.lib.sasb200_mlp_image_t_bytes(), dtype=torch.uint8,
                                 device=self.device)
        self._packed = None
        self._infer_out = None
        self._sync_bf16()
        self._scratch_n = 0
        # host flags of the training graphs: a queued replay may still set one
        # when its graph is gone
        self._refused = []

    # bf16 copies used by the kernels
    def _sync_bf16(self):
        """Refresh the bf16 copies from weights that were set on the current
        stream; in order with the work on self.stream and on the current one."""
        torch = self.torch
        current = torch.cuda.current_stream(self.device)
        self._wversion = getattr(self, "_wversion", 0) + 1
        if not hasattr(self, "Wb"):
            self.Wb = [torch.empty_like(w, dtype=torch.bfloat16) for w in self.W]
            self.WTb = [torch.empty_like(w.t(), dtype=torch.bfloat16,
                                         memory_format=torch.contiguous_format) for w in self.W]
        # in place: a captured training step holds their addresses, and kernels
        # on self.stream may still read or write them
        self.stream.wait_stream(current)
        with torch.cuda.stream(self.stream):
            for w, wb, wtb in zip(self.W, self.Wb, self.WTb):
                wb.copy_(w)
                wtb.copy_(w.t())
        current.wait_stream(self.stream)

    def _ptrs(self, tensors):
        arr = (ct.c_void_p*len(tensors))(*[t.data_ptr() for t in tensors])
        return arr

    def _check(self, status, what):
        if status != 0:
            raise RuntimeError("%s failed (%d): %s" % (what, status,
                                                      self.lib.sasb200_mlp_last_error().decode()))

    def _scratch(self, n_pad):
        torch = self.torch
        if n_pad <= self._scratch_n:
            return
        bf = dict(dtype=torch.bfloat16, device=self.device)
        f32 = dict(dtype=torch.float32, device=self.device)
        # planes of a training step (tiled) and of forward(save=True)
        self.z_save = torch.empty(4*n_pad*HID, **bf)
        self.h_save = torch.empty(4*n_pad*HID, **bf)
        self.dz_save = torch.empty(4*n_pad*HID, **bf)
        self.out = torch.empty(n_pad, **f32)
        self.dout = torch.empty(n_pad, **f32)
        self.row_sums = torch.empty(2*(n_pad//32), **f32)
        # gradients as partial sums over splits of the rows
        self.gW = [torch.empty(self.splits*HID*(NIN if l == 0 else HID), **f32)
                   for l in range(4)]
        self.gb_part = torch.empty((4, self.splits*HID), **f32)
        self.gw_part = torch.empty(self.splits*HID, **f32)
        self.gb = [torch.empty(HID, **f32) for _ in range(4)]
        self.gw = torch.empty(HID, **f32)
        self.gbo = torch.empty(1, **f32)
        # their addresses, which change with them only
        p = self._pass = _Pass(splits=self.splits, err=self.err.data_ptr())
        for field, t in (("z", self.z_save), ("h", self.h_save), ("dz", self.dz_save),
                         ("out", self.out), ("dout", self.dout), ("row_sums", self.row_sums),
                         ("db", self.gb_part), ("dw_out", self.gw_part)):
            setattr(p, field, t.data_ptr())
        p.dw[:] = [g.data_ptr() for g in self.gW]
        self._part_at = (list(p.dw) + [p.db + 4*self.splits*HID*l for l in range(4)]
                         + [p.dw_out])
        self._scratch_n = n_pad

    # ----------------------------------------------------------- kernels --
    def _pack(self):
        """Refresh the chunked weight image of the inference kernel after the
        bf16 weights changed (training steps, loads)."""
        key = (self.step_count, self._wversion)
        if self._packed == key:
            return
        self._pack_kernels()
        self._packed = key

    def _pack_kernels(self):
        self._check(self.lib.sasb200_mlp_pack(*[w.data_ptr() for w in self.Wb],
                                              self.img.data_ptr(), self.stream.cuda_stream),
                    "mlp_pack")
        self._check(self.lib.sasb200_mlp_pack_t(*[w.data_ptr() for w in self.WTb[1:]],
                                                self.img_t.data_ptr(), self.stream.cuda_stream),
                    "mlp_pack_t")

    def infer(self, x, x_lo, n, blocks=0):
        """Inference only: out[n_pad] for features x + x_lo through the
        persistent pipelined kernel (mlp_infer), on self.stream."""
        torch = self.torch
        n_pad = x.shape[0]
        if self._infer_out is None or self._infer_out.numel() < n_pad:
            self._infer_out = torch.empty(n_pad, dtype=torch.float32, device=self.device)
        self._pack()
        self._check(self.lib.sasb200_mlp_infer(
            n, n_pad, x.data_ptr(), x_lo.data_ptr(), self.img.data_ptr(), self._ptrs(self.b),
            self.w_out.data_ptr(), self.b_out.data_ptr(), self._infer_out.data_ptr(), None, None,
            self.err.data_ptr(), int(blocks), self.stream.cuda_stream), "mlp_infer")
        return self._infer_out[:n_pad]

    def serve(self, x, x_lo, n, blocks=0):
        """Inference only, through the overlapped kernel (mlp_serve): the
        hidden activations of :meth:`infer` with the output dot summed in
        another order; on self.stream."""
        torch = self.torch
        n_pad = x.shape[0]
        if self._infer_out is None or self._infer_out.numel() < n_pad:
            self._infer_out = torch.empty(n_pad, dtype=torch.float32, device=self.device)
        self._pack()
        self._check(self.lib.sasb200_mlp_serve(
            n, n_pad, x.data_ptr(), x_lo.data_ptr(), self.img.data_ptr(), self._ptrs(self.b),
            self.w_out.data_ptr(), self.b_out.data_ptr(), self._infer_out.data_ptr(), None, None,
            self.err.data_ptr(), int(blocks), self.stream.cuda_stream), "mlp_serve")
        return self._infer_out[:n_pad]

    def forward(self, x, x_lo, n, save=False):
        """out[n_pad] for features x + x_lo (bf16 [n_pad x 16] each), on
        self.stream."""
        n_pad = x.shape[0]
        self._scratch(n_pad)
        st = self.stream.cuda_stream
        w = self._ptrs(self.Wb)
        b = self._ptrs(self.b)
        self._check(self.lib.sasb200_mlp_forward(
            n, n_pad, x.data_ptr(), x_lo.data_ptr(), w, b, self.w_out.data_ptr(),
            self.b_out.data_ptr(),
            self.out.data_ptr(), self.z_save.data_ptr() if save else None,
            self.h_save.data_ptr() if save else None, self.err.data_ptr(), st), "mlp_forward")
        return self.out[:n_pad]

    def gradients(self, x, x_lo, y, n):
        """Loss and gradients of one batch, all on self.stream: returns
        (loss, dW split partials [4], db [4], dw_out, db_out)."""
        torch = self.torch
        self._scratch(x.shape[0])
        self._pack()
        with torch.cuda.stream(self.stream):
            loss = torch.empty((), dtype=torch.float32, device=self.device)
        self._gradient_kernels(x, x_lo, y, n, loss.data_ptr(), self.gbo.data_ptr(), 4,
                               [t.data_ptr() for t in self.gb + [self.gw]])
        return loss, self.gW, self.gb, self.gw, self.gbo

    def _gradient_kernels(self, x, x_lo, y, n, loss, db_out, first=9, outs=(), batch=None):
        """Forward, backward and weight gradients of one batch: the loss and
        db_out as scalars, the other gradients as partial sums over
        self.splits (gW, gb_part, gw_part); those of the parameters from
        `first` on (in the order of params, up to w_out) added over the splits
        into `outs`.  loss, db_out and outs are addresses.  With `batch` (a
        _Batch), x, x_lo and y receive its rows first."""
        p, sums = self._pass, len(outs)
        p.n, p.n_pad, p.delta = n, x.shape[0], float(self.huber)
        p.x, p.x_lo, p.y = x.data_ptr(), x_lo.data_ptr(), y.data_ptr()
        p.img, p.img_t = self.img.data_ptr(), self.img_t.data_ptr()
        p.b[:] = [t.data_ptr() for t in self.b]
        p.w_out, p.b_out = self.w_out.data_ptr(), self.b_out.data_ptr()
        p.loss, p.db_out, p.sums = loss, db_out, sums
        if sums:
            p.sum_sizes[:sums] = self._sizes[first:9]
            p.sum_splits[:sums] = [self.splits]*sums
            p.sum_parts[:sums] = self._part_at[first:]
            p.sum_outs[:sums] = outs
        p.batch = None if batch is None else ct.addressof(batch)
        self._check(self.lib.sasb200_mlp_train_pass(ct.byref(p), self.stream.cuda_stream),
                    "train_pass")

    def train_step(self, x, x_lo, y, n, lr, b1=0.9, b2=0.999, eps=1e-8, reduce=None):
        """One Adam step on one batch; returns the loss (a device scalar).

        `reduce`, when given, makes this a data-parallel step: it is called
        on self.stream with the list from `reduced_gradients` and must
        average it in place over the replicas (``multigpu.allreduce_mean``:
        one all-reduce of one flat bucket), after which every replica
        applies the same update."""
        if reduce is None:
            loss, dW, db, gw, gbo = self.gradients(x, x_lo, y, n)
            self.apply_gradients(dW + db + [gw, gbo], lr, self.splits, b1, b2, eps)
            return loss
        grads = self.reduced_gradients(x, x_lo, y, n)
        with self.torch.cuda.stream(self.stream):
            reduce(grads)
        self.apply_gradients(grads[1:], lr, 1, b1, b2, eps)
        return grads[0][0]

    def reduced_gradients(self, x, x_lo, y, n):
        """[loss (1 element), dW_1..dW_4, db_1..db_4, dw_out, db_out] of one
        batch as fp32 device tensors, the weight gradients summed over their
        partials: the ≈200k numbers a data-parallel step exchanges."""
        torch = self.torch
        self._scratch(x.shape[0])
        self._pack()
        sizes = self._sizes
        with torch.cuda.stream(self.stream):
            flat = torch.empty(sum(sizes) + 1, dtype=torch.float32, device=self.device)
        ends = [flat.data_ptr() + 4*sum(sizes[:k]) for k in range(len(sizes) + 1)]
        self._gradient_kernels(x, x_lo, y, n, ends[10], ends[9], 0, ends[:9])
        parts = flat.split(sizes + [1])
        return [parts[-1]] + list(parts[:-1])

    def capture_training(self, x_all, x_lo_all, y_all, batch, lr, total, step0, warmup=200,
                         b1=0.9, b2=0.999, eps=1e-8):
        """:class:`TrainingGraph` of one whole training step on `batch` rows
        of (x_all, x_lo_all, y_all) chosen by an index buffer, with the
        learning rate schedule of :meth:`Surrogate._train` (lr, total steps,
        linear warm-up over `warmup` steps, cosine decay) advancing on the
        device from schedule step `step0`."""
        return TrainingGraph(self, x_all, x_lo_all, y_all, batch, lr, total, step0, warmup,
                             b1, b2, eps)

    def apply_gradients(self, grads, lr, splits, b1=0.9, b2=0.999, eps=1e-8):
        """Adam update from [dW_1..dW_4 (each `splits` partials), db_1..db_4,
        dw_out, db_out], refreshing the bf16 weight copies; on self.stream."""
        self.step_count += 1
        self._adam(grads, [splits]*4 + [1]*6, None, lr, b1, b2, eps)
        # the update refreshed the weight images as well
        self._packed = (self.step_count, self._wversion)

    def _adam(self, grads, splits, sched, lr, b1, b2, eps):
        # the kernel reads the weights' gradients in 16-byte units
        with self.torch.cuda.stream(self.stream):
            grads = [g if k >= 4 or g.data_ptr() % 16 == 0 else g.clone()
                     for k, g in enumerate(grads)]
        self._check(self.lib.sasb200_adam_pack(
            self._ptrs(grads), (ct.c_int32*10)(*splits), self._ptrs(self.params),
            self._ptrs(self.m), self._ptrs(self.v), self._ptrs(self.Wb), self._ptrs(self.WTb),
            self.img.data_ptr(), self.img_t.data_ptr(),
            None if sched is None else sched.data_ptr(), lr, self.step_count, b1, b2, eps,
            self.stream.cuda_stream), "adam_pack")

    def features(self, radius, length, rpd, lpd, contrast, q, flag):
        """Compensated bf16 features (hi, lo) [n_pad x 16] on the device from
        float64 arrays (host arrays, or device tensors already on this
        network's stream)."""
        torch = self.torch
        n = len(q)
        n_pad = pad128(n)
        arrs = [a.contiguous() if isinstance(a, torch.Tensor) else
                torch.as_tensor(np.ascontiguousarray(a, 'd'), device=self.device)
                for a in (radius, length, rpd, lpd, contrast, q, flag)]
        x = torch.empty((n_pad, NIN), dtype=torch.bfloat16, device=self.device)
        x_lo = torch.empty((n_pad, NIN), dtype=torch.bfloat16, device=self.device)
        with torch.cuda.stream(self.stream):
            self._check(self.lib.sasb200_mlp_features(n, n_pad, *[a.data_ptr() for a in arrs],
                                                      x.data_ptr(), x_lo.data_ptr(),
                                                      self.stream.cuda_stream),
                        "features")
        return x, x_lo, n

    def errors(self):
        return int(self.err.item())

    def state(self):
        return {k: [t.detach().cpu().numpy() for t in v] if isinstance(v, list)
                else v.detach().cpu().numpy()
                for k, v in (("W", self.W), ("b", self.b), ("w_out", self.w_out),
                             ("b_out", self.b_out))}

    def load_state(self, st):
        """Set the weights (arrays or tensors ready on the current stream), behind
        the work queued on self.stream and ahead of what follows there."""
        torch = self.torch
        torch.cuda.current_stream(self.device).wait_stream(self.stream)
        for l in range(4):
            self.W[l].copy_(torch.as_tensor(st["W"][l]))
            self.b[l].copy_(torch.as_tensor(st["b"][l]))
        self.w_out.copy_(torch.as_tensor(st["w_out"]))
        self.b_out.copy_(torch.as_tensor(st["b_out"]).reshape(1))
        self._sync_bf16()


# --------------------------------------------------------------------------
# data, training, calibration and inference with fallback
# --------------------------------------------------------------------------

def sample_sets(n_sets, rng, flag=None, low_pd_frac=0.0, low_pd_max=0.08):
    """Parameter sets drawn over the training domain (log-uniform sizes,
    uniform polydispersities and contrast, random orientation flag).  With
    low_pd_frac > 0 that fraction of the sets draws its dispersities from
    [0, low_pd_max] instead, oversampling the sharply oscillating curves the
    network finds hardest."""
    lo, hi = DOMAIN["radius"]
    R = np.exp(rng.uniform(np.log(lo), np.log(hi), n_sets))
    lo, hi = DOMAIN["length"]
    L = np.exp(rng.uniform(np.log(lo), np.log(hi), n_sets))
    rpd = rng.uniform(*DOMAIN["rpd"], n_sets)
    lpd = rng.uniform(*DOMAIN["lpd"], n_sets)
    if low_pd_frac > 0:
        low = rng.uniform(0, 1, n_sets) < low_pd_frac
        rpd[low] = rng.uniform(0, low_pd_max, low.sum())
        lpd[low] = rng.uniform(0, low_pd_max, low.sum())
    contrast = rng.uniform(*DOMAIN["contrast"], n_sets)
    f = rng.integers(0, 2, n_sets) if flag is None else np.full(n_sets, flag)
    return dict(radius=R, length=L, rpd=rpd, lpd=lpd, contrast=contrast, flag=f)


def sample_q(nq, rng):
    lo, hi = DOMAIN["q"]
    return np.sort(np.exp(rng.uniform(np.log(lo), np.log(hi), nq)))


def model_pars(R, L, rpd, lpd, flag):
    """Parameters of the plain cylinder at unit contrast (scale 1, no
    background); dispersity 35 points over 3 sigma when the width is > 0."""
    p = dict(radius=float(R), length=float(L), sld=1.0, sld_solvent=0.0,
             scale=1.0, background=0.0)
    if rpd > 0:
        p.update(radius_pd=float(rpd), radius_pd_n=PD_N, radius_pd_nsigma=3.0)
    if lpd > 0:
        p.update(length_pd=float(lpd), length_pd_n=PD_N, length_pd_nsigma=3.0)
    if not flag:
        p.update(theta=90.0, phi=0.0)
    return p


def model_columns(sets, idx, flag):
    """`model_pars` of the sets `idx` as parameter columns (a width of 0
    leaves the parameter without dispersity, as model_pars omits it)."""
    cols = dict(radius=np.asarray(sets["radius"], float)[idx],
                length=np.asarray(sets["length"], float)[idx], sld=1.0, sld_solvent=0.0,
                scale=1.0, background=0.0,
                radius_pd=np.maximum(np.asarray(sets["rpd"], float)[idx], 0.0),
                radius_pd_n=PD_N, radius_pd_nsigma=3.0,
                length_pd=np.maximum(np.asarray(sets["lpd"], float)[idx], 0.0),
                length_pd_n=PD_N, length_pd_nsigma=3.0)
    if not flag:
        cols.update(theta=90.0, phi=0.0)
    return cols


def plain_unit_iq(sets, qs, device=None, form="float32c", shape=None):
    """I(q) at unit contrast from the plain engines, one array per set, both
    through the batched engine: flag 1 as the 1D orientation average, flag 0
    as the 2D kernel at theta = 90, phi = 0 along qx (the line form, equal
    to Iqxy at q vectors (q, 0))."""
    from .batch import Population
    n = len(qs)
    out = [None]*n
    pops = []
    # both populations are packed and enqueued before either is read back,
    # so the host packing of the second overlaps the first one's kernels
    flags = np.asarray(sets["flag"]).astype(bool)
    for flag in (1, 0):
        idx = np.nonzero(flags == bool(flag))[0]
        if not idx.size:
            continue
        warps, ipw = (shape or {}).get(flag, (8, 8))
        pop = Population.from_columns("cylinder", [qs[k] for k in idx],
                                      model_columns(sets, idx, flag), form=form,
                                      device=device, line=not flag, warps=warps,
                                      items_per_warp=ipw)
        pop.run()
        pops.append((idx, pop))
    for idx, pop in pops:
        for k, iq in zip(idx, pop.iq()):
            out[k] = iq.copy()
    return out


def flatten(sets, qs):
    """Flat per-point arrays of (set parameters, q); "set" is the index of
    the parameter set each point belongs to."""
    counts = np.array([len(q) for q in qs])
    cols = {key: np.repeat(np.asarray(sets[key]), counts)
            for key in ("radius", "length", "rpd", "lpd", "contrast", "flag")}
    cols["q"] = np.concatenate(qs)
    cols["set"] = np.repeat(np.arange(len(qs)), counts)
    return cols


def envelope(err, set_id, window):
    """Running maximum of err over the `window` neighbours on each side
    within the same set (points of a set contiguous and sorted by q): the
    local error envelope, smooth where err itself crosses zero."""
    env = np.array(err, dtype=float, copy=True)
    sid = np.asarray(set_id)
    for s in range(1, window + 1):
        same = sid[s:] == sid[:-s]
        np.maximum(env[s:], np.where(same, err[:-s], 0.0), out=env[s:])
        np.maximum(env[:-s], np.where(same, err[s:], 0.0), out=env[:-s])
    return env


def gate_thresholds(r, err, tols, alpha):
    """For each tolerance, the largest threshold t on the gate's predicted
    error r such that among the points with r <= t at most a fraction
    `alpha` have err > tolerance (0 if no threshold qualifies); made
    non-decreasing in the tolerance."""
    order = np.argsort(r, kind="stable")
    rs, es = np.asarray(r)[order], np.asarray(err)[order]
    k = np.arange(1, len(rs) + 1)
    out = []
    for tol in tols:
        fine = np.flatnonzero(np.cumsum(es > tol) <= alpha*k)
        out.append(rs[fine[-1]] if len(fine) else 0.0)
    return np.maximum.accumulate(np.array(out, dtype=float))


class TrainingGraph:
    """One training step of an :class:`MLP` captured as a CUDA graph: the
    batch gather (rows named by ``idx``) and the learning-rate schedule,
    forward and loss, backward, weight gradients, and Adam for every
    parameter with the bf16 weights and their images; the schedule's counters
    live on the device, so a replay needs only the new row indices."""

    def __init__(self, net, x_all, x_lo_all, y_all, batch, lr, total, step0, warmup,
                 b1, b2, eps):
        torch = net.torch
        self.net = net
        dev = net.device
        if batch % TM:
            raise ValueError("batch must be a multiple of %d" % TM)
        # the kernels take addresses
        if any(t.device != dev for t in (x_all, x_lo_all, y_all)):
            raise ValueError("the data set must be on %s" % dev)
        self.batch = batch
        self.idx = torch.zeros(batch, dtype=torch.int64, device=dev)
        self.counters = torch.tensor([int(step0), int(net.step_count)], dtype=torch.int32,
                                     device=dev)
        self.sched = torch.zeros(4, dtype=torch.float32, device=dev)
        self.xb = torch.empty((batch, x_all.shape[1]), dtype=x_all.dtype, device=dev)
        self.xlb = torch.empty_like(self.xb)
        self.yb = torch.empty(batch, dtype=y_all.dtype, device=dev)
        self.loss = torch.zeros((), dtype=torch.float32, device=dev)
        self._done = torch.cuda.Event()
        net._scratch(batch)
        lib, st = net.lib, net.stream.cuda_stream
        # the forward gathers 32-byte rows of bf16 and float targets, as
        # MLP.features (whose rows are padded to whole tiles) and the surrogate
        # lay them out
        direct = self.direct = (all(t.dtype == torch.bfloat16 and t.dim() == 2 and t.shape[1] == NIN
                      for t in (x_all, x_lo_all))
                  and y_all.dtype == torch.float32 and y_all.dim() == 1
                  and len(y_all) <= min(len(x_all), len(x_lo_all))
                  and all(t.is_contiguous() and t.data_ptr() % 16 == 0
                          for t in (x_all, x_lo_all, y_all)))
        rates = (int(total), int(warmup), float(lr), b1, b2)
        schedule = (self.counters.data_ptr(), self.sched.data_ptr())
        refused = torch.zeros(1, dtype=torch.int32).pin_memory()
        net._refused.append(refused)
        self._refused = refused.numpy()
        net.stream.synchronize()
        if net.errors() == ROW_OUTSIDE:
            net.err.zero_()          # of a graph before, which stays refused
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph, stream=net.stream):
            if not direct:
                torch.index_select(x_all, 0, self.idx, out=self.xb)
                torch.index_select(x_lo_all, 0, self.idx, out=self.xlb)
                torch.index_select(y_all, 0, self.idx, out=self.yb)
                net._check(lib.sasb200_lr_schedule(*schedule, *rates, st), "lr_schedule")
            net._gradient_kernels(
                self.xb, self.xlb, self.yb, batch, self.loss.data_ptr(), net.gbo.data_ptr(),
                batch=_Batch(self.idx.data_ptr(), len(y_all), x_all.data_ptr(), x_lo_all.data_ptr(),
                             y_all.data_ptr(), *schedule, refused.data_ptr(), *rates)
                if direct else None)
            net._adam(net.gW + list(net.gb_part) + [net.gw_part, net.gbo], [net.splits]*9 + [1],
                      self.sched, lr, b1, b2, eps)
        # what the graph reads and writes outlives the network's next, larger
        # scratch
        self._held = (x_all, x_lo_all, y_all, net.z_save, net.h_save, net.dz_save, net.out,
                      net.dout, net.row_sums, net.gW, net.gb_part, net.gw_part, net.gbo)

    def step(self, idx):
        """One training step on rows `idx` (int64 device tensor of `batch`
        entries); returns the loss (a device scalar, overwritten by the
        next step) for the current stream, which waits for the step.

        A row outside the data set ends the training of this graph, as it
        cannot be known before the kernels read it: the loss is NaN, weights
        and moments stay those of the step before, ``net.errors()`` is 5, and
        calls raise once the host has seen it."""
        net, torch = self.net, self.net.torch
        if self._refused[0]:
            raise RuntimeError(OUTSIDE)
        net._pack()          # current unless the weights were set from outside
        current = torch.cuda.current_stream(net.device)
        with torch.cuda.stream(net.stream):
            self.idx.copy_(idx)
            self.graph.replay()
        if current != net.stream:
            self._done.record(net.stream)
            current.wait_event(self._done)
        net.step_count += 1
        net._packed = (net.step_count, net._wversion)
        return self.loss


class Surrogate:
    """Trained network, its error gate, target scalings and the gate's
    calibrated thresholds."""

    TOL = 0.01
    #: tolerances (|log I error|) at which the gate is calibrated
    CAL_TOLS = np.unique(np.r_[np.logspace(-3, 0, 31), 0.01, 0.05])

    def __init__(self, device=None, seed=0):
        self.net = MLP(device=device, seed=seed)
        self.torch = self.net.torch
        self.seed = seed
        self.y_mean = 0.0
        self.y_std = 1.0
        self.gate = None
        self.g_mean = 0.0
        self.g_std = 1.0
        self.cal_tols = None
        self.cal_thresh = None
        self.alpha = None
        self.floor = 1e-5
        #: launch shape (warps, items per warp) of the batched fallback per
        #: orientation flag; None = the library default (8, 8)
        self.fallback_shape = None

    # ---- data --------------------------------------------------------------
    def dataset(self, n_sets, nq, seed, form="float32c", low_pd_frac=0.0):
        rng = np.random.default_rng(seed)
        sets = sample_sets(n_sets, rng, low_pd_frac=low_pd_frac)
        qs = [sample_q(nq, rng) for _ in range(n_sets)]
        iq = plain_unit_iq(sets, qs, self.net.device, form)
        cols = flatten(sets, qs)
        y = np.log(np.concatenate(iq))
        return cols, y

    def _x(self, cols):
        return self.net.features(cols["radius"], cols["length"], cols["rpd"], cols["lpd"],
                                 cols["contrast"], cols["q"], cols["flag"].astype(float))

    # ---- training ----------------------------------------------------------
    def _train(self, net, x_all, xlo_all, t_all, n, epochs, batch, lr, seed, scale, log, what,
               group=None):
        """Adam with cosine decay over shuffled batches of one network, all
        on its stream; returns the loss per epoch (in target units).

        Given a process group of several ranks (every rank holding the same
        training arrays and the same seed), each global batch is split into
        equal contiguous slices, one per rank, and the gradients averaged by
        one all-reduce per step: data-parallel replicas of the same run."""
        from .multigpu import allreduce_mean, batch_slice, broadcast_parameters
        torch = self.torch
        dist = torch.distributed
        nranks, rank, reduce = 1, 0, None
        if group is not None:
            nranks, rank = dist.get_world_size(group), dist.get_rank(group)
        if nranks > 1:
            broadcast_parameters(net, 0, group)

            def reduce(grads):
                allreduce_mean(grads, group)
        # the epochs' row orders come from a seeded generator on the device
        # (every replica of a data-parallel run draws the same ones)
        gen = torch.Generator(device=net.device)
        gen.manual_seed(int(seed))
        steps = max(1, n//batch)
        total = epochs*steps
        step = 0
        losses = []
        # on one GPU the first step runs eagerly (every kernel loaded), the
        # rest replay a CUDA graph of the step with the same schedule
        graph = None
        use_graph = nranks == 1 and (batch//nranks) % TM == 0
        for ep in range(epochs):
            perm = torch.randperm(n, device=net.device, generator=gen)
            net.stream.wait_stream(torch.cuda.current_stream(net.device))
            for s in range(steps):
                lo, hi = batch_slice(s*batch, batch, rank, nranks)
                idx = perm[lo:hi]
                if graph is not None:
                    loss = graph.step(idx)
                    step += 1
                    continue
                with torch.cuda.stream(net.stream):
                    xb = x_all.index_select(0, idx)
                    xlb = xlo_all.index_select(0, idx)
                    tb = t_all.index_select(0, idx)
                # cosine decay with a short warm-up
                frac = step/total
                rate = lr*min(1.0, (step + 1)/WARMUP_STEPS)*0.5*(1 + math.cos(math.pi*frac))
                loss = net.train_step(xb, xlb, tb, hi - lo, rate, reduce=reduce)
                step += 1
                if use_graph and step < total:
                    graph = net.capture_training(x_all, xlo_all, t_all, hi - lo, lr, total, step,
                                                 warmup=WARMUP_STEPS)
            net.stream.synchronize()
            losses.append(float(loss.item())*scale**2)
            if log:
                log("%s epoch %d loss %.3e" % (what, ep, losses[-1]))
        graph = None
        code = net.errors()
        if code:
            raise RuntimeError(OUTSIDE if code == ROW_OUTSIDE else
                               "tensor-core kernel reported a timeout")
        return losses

    def fit(self, cols, y, epochs=8, batch=8192, lr=2e-3, seed=0, log=None, huber=0.05,
            group=None):
        """Train the network on log I at unit contrast (Huber loss with
        threshold `huber` in log I); data-parallel over the ranks of
        `group` (e.g. ``torch.distributed.group.WORLD``) when given."""
        torch = self.torch
        good = np.isfinite(y)
        cols = {k: v[good] for k, v in cols.items()}
        y = y[good]
        self.y_mean = float(y.mean())
        self.y_std = float(y.std())
        self.net.huber = huber/self.y_std
        x_all, xlo_all, n = self._x(cols)
        t_all = torch.as_tensor((y - self.y_mean)/self.y_std, dtype=torch.float32,
                                device=self.net.device)
        return self._train(self.net, x_all, xlo_all, t_all, n, epochs, batch, lr, seed,
                           self.y_std, log, "net", group)

    def fit_gate(self, cols, y, epochs=16, batch=8192, lr=2e-3, seed=0, log=None, huber=1.0,
                 window=16, group=None):
        """Train the error gate: a second network of the same shape (the same
        tensor-core kernels) that predicts log(envelope + floor) of the
        trained network's |log I error| from the same features, on sets the
        network has not seen; the envelope is the running maximum over
        `window` neighbouring q of the set on each side (the error itself
        crosses zero between them, which no smooth predictor can follow).
        Returns the per-point errors."""
        torch = self.torch
        good = np.isfinite(y)
        cols = {k: v[good] for k, v in cols.items()}
        y = y[good]
        logi, _ = self._outputs(cols, gate=False)
        err = np.abs(logi - 2.0*np.log(np.abs(cols["contrast"])) - y)
        target = np.log(envelope(err, cols["set"], window) + self.floor)
        self.g_mean = float(target.mean())
        self.g_std = float(target.std())
        self.gate = MLP(device=self.net.device, seed=self.seed + 7919, stream=self.net.stream)
        self.gate.huber = huber/self.g_std
        x_all, xlo_all, n = self._x(cols)
        t_all = torch.as_tensor((target - self.g_mean)/self.g_std, dtype=torch.float32,
                                device=self.net.device)
        self._train(self.gate, x_all, xlo_all, t_all, n, epochs, batch, lr, seed + 1,
                    self.g_std, log, "gate", group)
        return err

    # ---- inference ----------------------------------------------------------
    def _outputs(self, cols, gate=True):
        """(predicted log I with the contrast, gate output or None) for flat
        arrays of inputs: one feature pass, both networks through the
        inference kernel."""
        torch = self.torch
        x, x_lo, n = self._x(cols)
        with torch.cuda.stream(self.net.stream):
            out = self.net.serve(x, x_lo, n)[:n].double()*self.y_std + self.y_mean
            g = None
            if gate and self.gate is not None:
                g = self.gate.serve(x, x_lo, n)[:n].double()*self.g_std + self.g_mean
            out = out.cpu()
            g = g.cpu() if g is not None else None
        self.net.stream.synchronize()
        logc = 2.0*np.log(np.abs(cols["contrast"]))
        return out.numpy() + logc, (g.numpy() if g is not None else None)

    def predict_log(self, cols):
        """Predicted log I (with the contrast) for flat arrays of inputs."""
        return self._outputs(cols, gate=False)[0]

    @staticmethod
    def inside(cols):
        """Points inside the training domain (with a nonzero contrast)."""
        ok = np.ones(len(cols["q"]), bool)
        for key in ("radius", "length", "rpd", "lpd", "contrast", "q"):
            lo, hi = DOMAIN[key]
            ok &= (cols[key] >= lo) & (cols[key] <= hi)
        return ok & (np.abs(cols["contrast"]) > 0)

    def _predicted(self, cols, g):
        """Smallest calibrated tolerance at which each point is accepted."""
        n = len(cols["q"])
        if g is None or self.cal_thresh is None:
            return np.full(n, np.inf)
        r = np.exp(g)
        # thresholds grow with the tolerance: first k with r <= thresh[k]
        k = np.searchsorted(self.cal_thresh, r, side="left")
        pe = np.where(k < len(self.cal_tols),
                      self.cal_tols[np.minimum(k, len(self.cal_tols) - 1)], np.inf)
        return np.where(self.inside(cols), pe, np.inf)

    def predicted_error(self, cols):
        """Predicted |log I error| per point: the smallest calibrated
        tolerance whose gate threshold admits the point; infinite outside the
        training domain or before calibration."""
        return self._predicted(cols, self._outputs(cols)[1])

    def calibrate(self, cols, y_true, alpha=5e-4):
        """Calibrate the gate on held-out sets judged by the plain FP64
        kernel: for each tolerance in CAL_TOLS, the largest threshold on
        exp(gate) for which at most a fraction `alpha` of the accepted
        points are in fact off by more than that tolerance.  Returns the
        per-point errors."""
        logi, g = self._outputs(cols)
        err = np.abs(logi - 2.0*np.log(np.abs(cols["contrast"])) - y_true)
        ok = self.inside(cols) & np.isfinite(err)
        self.cal_thresh = gate_thresholds(np.exp(g[ok]), err[ok], self.CAL_TOLS, alpha)
        self.cal_tols = self.CAL_TOLS.copy()
        self.alpha = alpha
        return err

    def _accept_log_threshold(self, tol):
        """log of the gate threshold at tolerance `tol` (the largest
        calibrated tolerance not above it); -inf when nothing is trusted."""
        if self.gate is None or self.cal_thresh is None:
            return -np.inf
        k = np.searchsorted(self.cal_tols, tol, side="right") - 1
        if k < 0 or self.cal_thresh[k] <= 0:
            return -np.inf
        return float(np.log(self.cal_thresh[k]))

    def _device_eval(self, cols, tol):
        """(I, accepted mask) of the network at every point, computed on the
        device: only q and one row per run of points sharing a parameter set
        cross to the GPU (points of a set are contiguous, as flatten() lays
        them out); the gate threshold and exp(log I) run there too."""
        torch = self.torch
        net, dev = self.net, self.net.device
        sid = np.asarray(cols["set"])
        n = len(sid)
        q = np.ascontiguousarray(cols["q"], 'd')
        # the kernels take addresses: q has a value for each of the n points
        if sid.ndim != 1 or q.shape != sid.shape:
            raise ValueError("q has shape %s, set %s" % (q.shape, sid.shape))
        if n == 0:
            return np.zeros(0), np.zeros(0, bool)
        starts = np.concatenate([[0], np.flatnonzero(sid[1:] != sid[:-1]) + 1])
        keys = ("radius", "length", "rpd", "lpd", "contrast", "flag")
        runs = len(starts)
        # one upload for the rows and, behind them, the runs' first points
        table = np.zeros((runs, 8))
        for j, k in enumerate(keys):
            table[:, j] = np.asarray(cols[k])[starts]
        ok = np.abs(table[:, 4]) > 0
        for j, key in enumerate(keys[:5]):
            lo, hi = DOMAIN[key]
            ok &= (table[:, j] >= lo) & (table[:, j] <= hi)
        table[:, 6] = ok
        rows = np.concatenate([table[:, :7].ravel(),
                               np.pad(starts, (0, runs % 2)).astype(np.int32).view(float)])
        thr = self._accept_log_threshold(tol)
        qlo, qhi = DOMAIN["q"]
        n_pad = pad128(n)
        with torch.cuda.stream(net.stream):
            rows = torch.as_tensor(rows, device=dev)
            q = torch.as_tensor(q, device=dev)
            feats = torch.empty((2, n_pad, NIN), dtype=torch.bfloat16, device=dev)
            result = torch.empty(n + (n + 7)//8, dtype=torch.float64, device=dev)
            st = net.stream.cuda_stream
            table_ptr = rows.data_ptr()
            starts_ptr = table_ptr + 8*7*runs
            x, x_lo = feats[0], feats[1]
            net._check(net.lib.sasb200_features_runs(
                n, n_pad, runs, starts_ptr, table_ptr, q.data_ptr(), x.data_ptr(),
                x_lo.data_ptr(), st), "features_runs")
            out = net.serve(x, x_lo, n)
            g = self.gate.serve(x, x_lo, n) if np.isfinite(thr) else None
            net._check(net.lib.sasb200_finish_runs(
                n, runs, starts_ptr, table_ptr, q.data_ptr(), out.data_ptr(),
                None if g is None else g.data_ptr(), self.y_std, self.y_mean, self.g_std,
                self.g_mean, thr, qlo, qhi, result.data_ptr(), result.data_ptr() + 8*n, st),
                "finish_runs")
            host = result.cpu().numpy()
        return host[:n], host[n:].view(np.bool_)[:n]

    def iq(self, cols, tol=None, device=None, form="float32c"):
        """I(q) for flat inputs: the network where its predicted error is
        within `tol` (log I), the plain kernel elsewhere (its FP32c form by
        default, within 1e-5 of FP64, far inside the tolerance).  Returns
        (I, mask of points that fell back)."""
        tol = self.TOL if tol is None else tol
        I, accepted = self._device_eval(cols, tol)
        back = ~accepted
        if back.any():
            I[back] = self.plain(cols, back, device, form)
        return I, back

    def plain(self, cols, mask, device=None, form="double"):
        """Plain-kernel I(q) (with contrast) at the masked points, one plain
        evaluation per parameter set over just its masked q."""
        idx = np.nonzero(mask)[0]
        sid = cols["set"][idx]
        order = np.argsort(sid, kind="stable")
        idx, sid = idx[order], sid[order]
        starts = np.flatnonzero(np.r_[True, sid[1:] != sid[:-1]])
        ends = np.r_[starts[1:], len(sid)]
        first = idx[starts]
        sets = {k: cols[k][first] for k in ("radius", "length", "rpd", "lpd", "contrast",
                                            "flag")}
        sets["flag"] = sets["flag"].astype(int)
        qs = [cols["q"][idx[a:b]] for a, b in zip(starts, ends)]
        iq = plain_unit_iq(sets, qs, device or self.net.device, form,
                           shape=self.fallback_shape if form == "float32c" else None)
        vals = np.empty(len(idx))
        for (a, b), v, c in zip(zip(starts, ends), iq, sets["contrast"]):
            vals[a:b] = v*c*c
        out = np.empty(len(mask))
        out[idx] = vals
        return out[mask]

    def save(self, path):
        st = self.net.state()
        extra = {}
        if self.gate is not None:
            gs = self.gate.state()
            extra = dict(**{"gW%d" % l: gs["W"][l] for l in range(4)},
                         **{"gb%d" % l: gs["b"][l] for l in range(4)},
                         g_w_out=gs["w_out"], g_b_out=gs["b_out"])
        if self.cal_thresh is not None:
            extra.update(cal_tols=self.cal_tols, cal_thresh=self.cal_thresh)
        np.savez(path, y_mean=self.y_mean, y_std=self.y_std, g_mean=self.g_mean,
                 g_std=self.g_std, floor=self.floor,
                 **{"W%d" % l: st["W"][l] for l in range(4)},
                 **{"b%d" % l: st["b"][l] for l in range(4)},
                 w_out=st["w_out"], b_out=st["b_out"], **extra)

    def load(self, path):
        d = np.load(path)
        self.y_mean = float(d["y_mean"])
        self.y_std = float(d["y_std"])
        self.net.load_state({"W": [d["W%d" % l] for l in range(4)],
                             "b": [d["b%d" % l] for l in range(4)],
                             "w_out": d["w_out"], "b_out": d["b_out"]})
        if "gW0" in d:
            self.g_mean, self.g_std = float(d["g_mean"]), float(d["g_std"])
            self.floor = float(d["floor"])
            self.gate = MLP(device=self.net.device, seed=self.seed + 7919,
                            stream=self.net.stream)
            self.gate.load_state({"W": [d["gW%d" % l] for l in range(4)],
                                  "b": [d["gb%d" % l] for l in range(4)],
                                  "w_out": d["g_w_out"], "b_out": d["g_b_out"]})
        if "cal_thresh" in d:
            self.cal_tols, self.cal_thresh = d["cal_tols"], d["cal_thresh"]


def train_and_evaluate(n_train_sets=50000, nq=1000, epochs=10, n_holdout_sets=1000,
                       batch=8192, lr=2e-3, tol=0.01, seed=0, device=None, log=None,
                       data_form="float32c", low_pd_frac=0.4, n_gate_sets=None,
                       gate_epochs=16, alpha=5e-4):
    """
    Generate training data with the plain kernels and train the network;
    train the error gate on fresh sets; on held-out sets judged by the plain
    FP64 kernels, calibrate the gate thresholds (two thirds) and measure (one
    third): accuracy, and the throughput of the surrogate with automatic
    fallback against the plain FP64 (and FP32c) path on the same points.
    """
    import time
    import torch
    say = log or (lambda *a: None)
    S = Surrogate(device=device, seed=seed)
    t0 = time.perf_counter()
    cols, y = S.dataset(n_train_sets, nq, seed + 1, form=data_form, low_pd_frac=low_pd_frac)
    torch.cuda.synchronize()
    t_data = time.perf_counter() - t0
    say("data: %d samples in %.1f s" % (len(y), t_data))
    t0 = time.perf_counter()
    losses = S.fit(cols, y, epochs=epochs, batch=batch, lr=lr, seed=seed, log=say)
    torch.cuda.synchronize()
    t_train = time.perf_counter() - t0
    del cols, y
    # error gate on sets the network has not seen (FP32c labels: within 1e-5,
    # far inside the tolerances)
    if n_gate_sets is None:
        n_gate_sets = max(n_train_sets//5, 300)
    t0 = time.perf_counter()
    gcols, gy = S.dataset(n_gate_sets, nq, seed + 3, form=data_form, low_pd_frac=low_pd_frac)
    S.fit_gate(gcols, gy, epochs=gate_epochs, batch=batch, lr=lr, seed=seed, log=say)
    torch.cuda.synchronize()
    t_gate = time.perf_counter() - t0
    del gcols, gy
    rng = np.random.default_rng(seed + 2)
    sets = sample_sets(n_holdout_sets, rng)
    qs = [sample_q(nq, rng) for _ in range(n_holdout_sets)]
    half = (2*n_holdout_sets)//3
    cal = ({k: v[:half] for k, v in sets.items()}, qs[:half])
    ev = ({k: v[half:] for k, v in sets.items()}, qs[half:])
    cal_cols = flatten(*cal)
    cal_y = np.log(np.concatenate(plain_unit_iq(cal[0], cal[1], S.net.device, "double")))
    S.calibrate(cal_cols, cal_y, alpha=alpha)
    ev_cols = flatten(*ev)
    # plain FP64 path on the measured part (also the ground truth), and the
    # plain FP32c path for reference; one untimed call of each first
    plain_unit_iq({k: v[:8] for k, v in ev[0].items()}, ev[1][:8], S.net.device, "double")
    plain_unit_iq({k: v[:8] for k, v in ev[0].items()}, ev[1][:8], S.net.device, "float32c")
    # every arm below is timed on the host clock as the mean of REPS calls,
    # so that one stall of the host does not decide a ratio
    REPS = 3

    def timed(fn):
        out, total = None, 0.0
        for _ in range(REPS):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            out = fn()
            torch.cuda.synchronize()
            total += time.perf_counter() - t0
        return out, total/REPS
    ev_iq, t_plain = timed(lambda: plain_unit_iq(ev[0], ev[1], S.net.device, "double"))
    _, t_plain32 = timed(lambda: plain_unit_iq(ev[0], ev[1], S.net.device, "float32c"))
    truth = np.log(np.concatenate(ev_iq)) + 2*np.log(np.abs(ev_cols["contrast"]))
    S.predict_log(ev_cols)            # warm
    _, t_net = timed(lambda: S.predict_log(ev_cols))
    logi, g = S._outputs(ev_cols)
    raw = np.abs(logi - truth)
    n = len(truth)
    report = dict(
        train_samples=int(n_train_sets*nq), epochs=epochs, data_s=t_data, train_s=t_train,
        gate_samples=int(n_gate_sets*nq), gate_epochs=gate_epochs, gate_s=t_gate,
        gate_alpha=alpha, final_loss=losses[-1], holdout_samples=int(n),
        net_median_err=float(np.median(raw)), net_p90_err=float(np.quantile(raw, 0.9)),
        net_p99_err=float(np.quantile(raw, 0.99)),
        plain_samples_per_s=n/t_plain, plain_f32c_samples_per_s=n/t_plain32,
        net_only_samples_per_s=n/t_net,
        net_only_speedup=t_plain/t_net, operating_points={})
    # surrogate with automatic fallback, timed end to end, at each tolerance
    # (one untimed call of each first: module loading, allocator warm-up)
    for t in sorted({tol, 0.05}):
        S.iq(ev_cols, tol=t)
    for t in sorted({tol, 0.05}):
        (I, back), t_sur = timed(lambda: S.iq(ev_cols, tol=t))
        err = np.abs(np.log(I) - truth)
        report["operating_points"]["%g" % t] = dict(
            net_frac_within=float(np.mean(raw <= t)), fallback_frac=float(back.mean()),
            frac_within=float(np.mean(err <= t)),
            accepted_frac_within=float(np.mean(err[~back] <= t)) if (~back).any() else 1.0,
            max_err=float(err.max()), samples_per_s=n/t_sur, speedup=t_plain/t_sur,
            speedup_vs_plain_f32c=t_plain32/t_sur)
    return S, report
