"""Backward pass of KNNConv on the tensor cores.

Both gradient contractions of ``out[b,o,n] = sum_k sum_c Xpad[b,c,idx[k,n]] * W[o, c*V + tap[n,k]]``
(fovi/arch/knn.py:538-557; the reference gets them from autograd through its gather, one-hot matmul and linear) are
themselves table-driven gather-GEMMs:

* input gradient — a forward launch of ``fovi_knnconv_forward`` on a derived plan, the transposed layer: "output" points are the layer's input points m, the neighbours of m are the
  output points n that list m, each with the tap it was given; channels swap roles
  (``dX[b,m,c] = sum_{(n,k): idx[k,n]=m} sum_o dY[b,n,o] * W[o, c*V + tap[n,k]]``).
* weight gradient — the contraction runs over the batch, one product [c_out x c_in] per (output point, neighbour) pair, summed per filter tap
  (``dW[o,c,v] = sum_{(n,k): tap[n,k]=v} sum_b dY[b,n,o] * X[b,idx[k,n],c]``).  A kernel of its own (``csrc/knnconv_dw.cu``) reads both operands in the
  layout the forward pass left them in: channels last (parts of a tap added in no fixed order, so repeated runs agree to float32 rounding), or the
  pair layout of a first layer with at most 4 channels (added in a fixed order: the same bits every time).

Operands are bf16 with float32 accumulation, as under the reference's autocast training.  Layers that run on the exact
float32 kernel (``precision='fp32'``, or shapes outside the tensor-core kernel) take the same two derived layers through
that kernel instead (``input_grad_f32`` / ``weight_grad_f32``): float32 arithmetic throughout, for parity work, not speed.
"""
import numpy as np
import torch

from . import ops

__all__ = ["KnnConvGrad", "knnconv_autograd", "knnconv_points_autograd", "block_autograd"]

MAX_LIST = 256      # longest neighbour list the tensor-core kernel takes


def _grouped(keys, n_groups, limit=None):
    """Stable grouping of entry indices by key.  Returns (order, group id of each ordered entry, position inside its
    group, number of groups, parts).  With `limit`, groups longer than it are cut into consecutive parts; `parts` is then
    either an int P (every key has P parts, some possibly empty: part p of key g is group g*P + p) or, when that would
    leave too many empty parts, the array of each group's owner key."""
    order = np.argsort(keys, kind="stable")
    k = keys[order]
    start = np.searchsorted(k, np.arange(n_groups))
    pos = np.arange(k.size) - start[k]
    if limit is None:
        return order, k, pos, n_groups, 1
    counts = np.bincount(k, minlength=n_groups)
    need = np.maximum(1, -(-counts // limit))
    P = int(need.max()) if need.size else 1
    if n_groups * P <= 1.3 * need.sum():                    # few empty parts: uniform, the parts are summed by a reduction
        return order, k * P + pos // limit, pos % limit, n_groups * P, P
    first = np.concatenate([[0], np.cumsum(need)[:-1]])     # uneven lists: as many parts as each key needs, summed by index
    return order, first[k] + pos // limit, pos % limit, int(need.sum()), np.repeat(np.arange(n_groups), need)


class KnnConvGrad:
    """Derived plans of one KNNConv layer's backward pass (built on first use, cached)."""

    def __init__(self, knn_idx_pad, tap, n_in, V, c_in, c_out, device):
        idx = np.asarray(knn_idx_pad).astype(np.int64)          # [K, n_out], pad == n_in
        tp = np.asarray(tap).astype(np.int64)                   # [n_out, K]
        self.n_in, self.V, self.c_in, self.c_out, self.device = int(n_in), int(V), int(c_in), int(c_out), device
        self.K, self.n_out = idx.shape
        ks, ns = np.nonzero(idx != n_in)
        self._n, self._m, self._v, self._k = ns, idx[ks, ns], tp[ns, ks], ks
        self._dx_plan = None
        self._dw_plans = {}
        self.cin_packed = self.c_in if self.c_in % 64 == 0 else -(-self.c_in // 8) * 8

    def check(self):
        """Synchronise the current stream and raise if a launch of the backward pass gave up on a wait (its gradient is incomplete).  A pair-layout
        layer's weight gradient reports through the layer's own plan."""
        for plan in [self._dx_plan] + [p for key, plans in self._dw_plans.items() for p in (plans[:1] if key == "dw" else plans[:2])]:
            if plan is not None:
                plan.check()

    # ---- dX
    def dx_plan(self):
        if self._dx_plan is None:
            if self.c_in % 16:
                raise NotImplementedError("input gradient needs in_channels to be a multiple of 16 (a first layer's input needs none)")
            order, gid, pos, _, _ = _grouped(self._m, self.n_in)
            kt = max(8, int(pos.max()) + 1 if pos.size else 8)
            if kt > MAX_LIST:
                raise NotImplementedError(f"an input point feeds {kt} outputs; the kernel takes lists up to {MAX_LIST}")
            idx_t = np.full((kt, self.n_in), self.n_out, np.int32)
            tap_t = np.zeros((self.n_in, kt), np.uint16)
            idx_t[pos, gid] = self._n[order]
            tap_t[gid, pos] = self._v[order]
            self._dx_plan = ops.KnnConvPlan(idx_t, tap_t, self.n_out, self.V, self.c_out, self.c_in, device=self.device)
            if not self._dx_plan.tc_supported:
                raise NotImplementedError("the transposed layer is outside the tensor-core kernel's shapes")
        return self._dx_plan

    def input_grad(self, gy_points, weight):
        """gy_points [B, n_out, c_out] bf16 contiguous, weight [c_out, c_in*V] -> dX [B, n_in, c_in] bf16 (channels last)."""
        plan = self.dx_plan()
        return plan.forward(gy_points, plan.pack_weights_transposed(weight), out_dtype=torch.bfloat16)

    def input_grad_masked(self, gy_points, weight, act):
        """`input_grad` of a layer whose input `act` [B, n_in, c_in] is a ReLU's result: (the gradient behind the mask, its sums per channel), or None."""
        plan = self.dx_plan()
        return plan.input_grad_masked(gy_points, plan.pack_weights_transposed(weight), act) if plan.masks_input_grad(gy_points.shape[0]) else None

    def masking_pays(self, rows):
        """Whether `input_grad_masked` is the faster form.  Per 64 columns of a tile (256 rows of an input point) the masked epilogue takes 2.0 us against 0.85, hidden behind
        the products of the next tile where there are enough; the separate pass costs by the row.  So the masked form loses where the last tile of rows is mostly
        empty AND a tile has few products: 129 rows, 1000 points: 512 <- 64 channels, 1 neighbour 170 -> 202 us, 9 neighbours 198 -> 218, 25 neighbours
        gains; 300 rows 340 -> 380; 256 rows 233 -> 224; grids of a few hundred tiles gain at any fill."""
        tiles, columns = -(-rows // 256), -(-self.c_in // 256)                    # row tiles; column tiles (of at most 256)
        products = self._n.size / self.n_in * -(-self.c_out // 64)
        return 3 * rows >= 2 * 256 * tiles or self.n_in * columns * tiles <= 700 or products >= 3 * (-(-self.c_in // (64 * columns)))

    # ---- dW
    @property
    def dw_swapped(self):
        """Which operand gives the rows of the weight-gradient products.  Rows come in tiles of 256 on a CTA pair or 128 on one CTA; a layer
        with few input and many output channels (64 -> 192) wastes less with the input's channels as rows."""
        return self.cin_packed <= 128 < self.c_out

    def dw_plan(self):
        """(plan, result row of each group).  A tap's pairs, sorted by output point, are cut into parts, a few hundred in all (several per CTA
        pair), and the parts of all taps are ordered by position: products that run at the same time then share points in L2 (tap by tap, every tap
        sweeps all of both operands: 2.5 GB from DRAM where they hold 0.3)."""
        if "dw" not in self._dw_plans:
            order = np.lexsort((self._m, self._n, self._v))
            v, n, m = self._v[order], self._n[order], self._m[order]
            limit = int(max(8, -(-v.size // 250)))
            start = np.searchsorted(v, np.arange(self.V + 1))
            groups = []
            for t in range(self.V):
                lo, hi = int(start[t]), int(start[t + 1])
                parts = -(-(hi - lo) // limit)
                groups += [(t, lo + (hi - lo) * i // parts, lo + (hi - lo) * (i + 1) // parts) for i in range(parts)]
            groups.sort(key=lambda g: (int(n[(g[1] + g[2]) // 2]), g[0]))
            kw = max([g[2] - g[1] for g in groups], default=1)
            pts, qts = (m, n) if self.dw_swapped else (n, m)
            p_pt, q_pt = np.zeros((max(1, len(groups)), kw), np.int32), np.zeros((max(1, len(groups)), kw), np.int32)
            cnt, owner = np.zeros(max(1, len(groups)), np.int32), np.zeros(max(1, len(groups)), np.int32)
            for i, (t, lo, hi) in enumerate(groups):
                p_pt[i, :hi - lo], q_pt[i, :hi - lo], cnt[i], owner[i] = pts[lo:hi], qts[lo:hi], hi - lo, t
            n_p, n_q = (self.n_in, self.n_out) if self.dw_swapped else (self.n_out, self.n_in)
            self._dw_plans["dw"] = (ops.KnnDwPlan(p_pt, q_pt, cnt, owner, self.V, n_p, n_q, self.device), owner)
        return self._dw_plans["dw"]

    def weight_grad(self, gy_points, x_points, plan, dtype=torch.float32):
        """gy_points [B, n_out, c_out] bf16 contiguous, x_points the layer's packed input ([B, n_in, cin_packed] bf16, or the pair layout with zero
        pad rows), plan the layer's own -> dW [c_out, c_in*V] (summed in float32)."""
        if plan.x_layout == ops.X_PAIRS:
            return ops.weight_grad_unpack(plan.weight_grad_pairs(gy_points, x_points), self.c_out, self.c_in, dtype=dtype)
        p, q = (x_points, gy_points) if self.dw_swapped else (gy_points, x_points)
        return ops.weight_grad(self.dw_plan()[0], p, q, self.c_out, self.c_in, self.dw_swapped, dtype)

    # ---- exact float32 route (precision='fp32' layers and shapes outside the tensor-core kernel): the same two derived
    # layers, run on the exact float32 kernel (fovi_knnconv_forward_f32) instead of the tensor cores
    def _f32_plans(self, B):
        key = ("f32", B)
        if key not in self._dw_plans:
            order, gid, pos, _, _ = _grouped(self._m, self.n_in)
            kt = max(1, int(pos.max()) + 1 if pos.size else 1)
            idx_t = np.full((kt, self.n_in), self.n_out, np.int32)
            tap_t = np.zeros((self.n_in, kt), np.uint16)
            idx_t[pos, gid] = self._n[order]
            tap_t[gid, pos] = self._v[order]
            dx = ops.KnnConvPlan(idx_t, tap_t, self.n_out, self.V, self.c_out, self.c_in, device=self.device)
            order, gid, pos, n_groups, parts = _grouped(self._v, self.V, 512)
            kw = max(1, int(pos.max()) + 1 if pos.size else 1)
            idx_w = np.full((kw, n_groups), self.n_out, np.int32)
            tap_w = np.zeros((n_groups, kw), np.uint16)
            idx_w[pos, gid] = self._n[order]
            tap_w[gid, pos] = self._m[order]
            dw = ops.KnnConvPlan(idx_w, tap_w, self.n_out, self.n_in, B, self.c_in, device=self.device)
            owner = np.arange(n_groups) // parts if isinstance(parts, int) else parts
            self._dw_plans[key] = (dx, dw, torch.from_numpy(np.ascontiguousarray(owner, dtype=np.int64)).to(self.device))
        return self._dw_plans[key]

    def input_grad_f32(self, gy, weight):
        """gy [B, c_out, n_out], weight [c_out, c_in*V] -> dX [B, c_in, n_in], float32 arithmetic throughout."""
        dx, _, _ = self._f32_plans(gy.shape[0])
        w_t = weight.detach().float().reshape(self.c_out, self.c_in, self.V).permute(1, 0, 2).reshape(self.c_in, self.c_out * self.V)
        return dx.forward_f32(gy.float(), dx.pack_weights(w_t.contiguous(), dtype=torch.float32))

    def weight_grad_f32(self, gy, x):
        """gy [B, c_out, n_out], x [B, c_in, n_in] -> dW [c_out, c_in*V] float32: rows = output channels, "channels" = the
        batch, "taps" = the input points holding X^T, one pseudo output point per part of a filter tap's pair list."""
        B = gy.shape[0]
        _, dw, owner = self._f32_plans(B)
        rows = gy.float().permute(1, 0, 2).contiguous()                               # [c_out, B, n_out]
        taps = torch.zeros((self.n_in, self.c_in, dw.cin_packed), dtype=torch.float32, device=gy.device)
        taps[:, :, :B] = x.float().permute(2, 1, 0)                                   # [n_in, c_in, B]
        parts = dw.forward_f32(rows, taps)                                            # [c_out, c_in, parts]
        out = torch.zeros((self.c_out, self.c_in, self.V), dtype=torch.float32, device=gy.device)
        out.index_add_(2, owner, parts)
        return out.reshape(self.c_out, self.c_in * self.V)


def _aligned(t):
    """The contiguous tensor t, copied if it does not start on the 16 bytes that the kernels' tensor copies need (an upstream gradient may be a piece
    of a larger buffer, as the backward of a concatenation hands out)."""
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _channels_last(t):
    """[B, C, N] of any strides and alignment -> contiguous, 16-byte aligned [B, N, C] bf16."""
    p = t.permute(0, 2, 1)
    if p.is_contiguous():
        return _aligned(p.to(torch.bfloat16))
    return ops.pack_points(t, t.shape[1]) if t.shape[1] % 8 == 0 else p.to(torch.bfloat16).contiguous()


class _KnnConvFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias, layer):
        ctx.layer = layer
        ctx.has_bias = bias is not None
        ctx.x_dtype = x.dtype
        ctx.f32 = layer.precision == "fp32" or not layer.plan.tc_supported       # the forward runs on the exact float32 kernel
        with torch.no_grad():
            if ctx.f32:
                ctx.save_for_backward(x, weight)
                return layer._forward(x)
            y, xp = layer._forward_packed(x)
        ctx.save_for_backward(xp if ctx.needs_input_grad[1] else None, weight)   # the packed input is all the weight gradient reads
        return y

    @staticmethod
    def backward(ctx, gy):
        x, weight = ctx.saved_tensors
        g = ctx.layer.grad_plans
        gx = gw = gb = None
        if ctx.f32:
            if ctx.needs_input_grad[0]:
                gx = g.input_grad_f32(gy, weight).to(x.dtype)
            if ctx.needs_input_grad[1]:
                gw = g.weight_grad_f32(gy, x).to(weight.dtype)
        elif ctx.needs_input_grad[0] or ctx.needs_input_grad[1]:
            gyp = _channels_last(gy)
            if ctx.needs_input_grad[0]:
                gx = g.input_grad(gyp, weight).permute(0, 2, 1).to(ctx.x_dtype)
            if ctx.needs_input_grad[1]:
                gw = g.weight_grad(gyp, x, ctx.layer.plan, weight.dtype)
        if ctx.has_bias and ctx.needs_input_grad[2]:
            gb = gy.sum((0, 2), dtype=torch.float32)
        return gx, gw, gb, None


def _mark(grad, link, sums):
    """Note on the gradient tensor itself that it is masked for the layer behind `link`, with its sums per channel.  (On the tensor, not in an object that the
    two layers share: two passes over one graph run their nodes in any order.)  An inference tensor counts no writes, so it carries no mark."""
    if not grad.is_inference():
        grad._fovi_masked = (link, grad._version, sums)


def _take_mark(grad, link):
    """The sums that `_mark` left on this gradient for this link, or None, also if it was written to since.  Whoever takes them owns them."""
    mark = grad.__dict__.pop("_fovi_masked", None)
    return mark[2] if mark is not None and link is not None and mark[0] is link and mark[1] == grad._version else None


class _KnnConvPointsFunction(torch.autograd.Function):
    """A layer on the kernels' own activation layout (channels last, bf16) with the ReLU fused, so that a chain of layers
    trains without a layout change between them.  `x` is [B, n_in, c_in] bf16, or for a pair-layout first layer the
    [B, c_in, n_in] input itself (it is packed here).

    `below` / `above`: objects that the layer shares with the one whose ReLU result is its input / whose input its ReLU result is, when nothing else reads
    it.  A layer's input gradient then leaves its kernel behind the mask of the layer below, and the sums of it, the bias gradient of that layer, travel ON the
    gradient tensor (`_mark`, `_take_mark`): the pass over the gradient that does both otherwise is left out (the mask is the same, zero or one: the gradient's
    bits are too).  A gradient that is not that tensor, or was written to since (by a hook on a node in between), takes that pass, which leaves a
    masked gradient as it is; such a hook sees the gradient behind the mask."""

    @staticmethod
    def forward(ctx, x, weight, bias, layer, relu, below=None, above=None):
        plan = layer.plan
        first = plan.x_layout == ops.X_PAIRS
        rows = x.shape[0]
        with torch.no_grad():
            xp = ops.pack_points(x, plan) if first else x.contiguous()
            y = plan.forward(xp, layer.packed_weight(), bias, relu=relu, out_dtype=torch.bfloat16, batch=rows)
        ctx.layer, ctx.relu, ctx.first, ctx.has_bias, ctx.below, ctx.above = layer, relu, first, bias is not None, below, above
        ctx.save_for_backward(xp if ctx.needs_input_grad[1] or (below is not None and ctx.needs_input_grad[0]) else None, weight, y if relu else None)
        return y

    @staticmethod
    def backward(ctx, gy):
        xp, weight, y = ctx.saved_tensors
        g = ctx.layer.grad_plans
        gb = _take_mark(gy, ctx.above)                     # there: gy is masked, and these are its sums
        gy = _aligned(gy.to(torch.bfloat16).contiguous())
        want_w, want_b = ctx.needs_input_grad[1], ctx.has_bias and ctx.needs_input_grad[2]
        if ctx.relu and gb is None:
            fused = ops.relu_mask_colsum(gy, y)            # mask and bias sums in one pass over the gradient
            if fused is not None:
                gy, gb = fused
            else:
                gy = torch.ops.aten.threshold_backward(gy, y, 0).contiguous()       # gy where y > 0, else 0
        gx = gw = None
        if ctx.needs_input_grad[0]:
            if ctx.first:
                raise NotImplementedError("input gradient of a pair-layout first layer is not built")
            both = g.input_grad_masked(gy, weight, xp) if ctx.below is not None and g.masking_pays(gy.shape[0]) else None
            if both is not None:
                gx, sums = both
                _mark(gx, ctx.below, sums)
            else:
                gx = g.input_grad(gy, weight)                                  # [B, n_in, c_in] bf16
        if want_w:
            gw = g.weight_grad(gy, xp, ctx.layer.plan, weight.dtype)
        if not want_b:
            gb = None
        elif gb is None:
            gb = ops.column_sum(gy) if gy.shape[-1] % 2 == 0 else gy.sum((0, 1), dtype=torch.float32)
        return gx, gw, gb, None, None, None, None


class _BlockFunction(torch.autograd.Function):
    """A block's convolution, training-mode batch norm, ReLU and max pooling (fovi/arch/knnalexnet.py:109-127).  The norm's forward pass is the module's own
    (`torch._batch_norm_impl_index`, which torch's batch_norm calls), so the activations are those of the separate modules bit for bit; what surrounds it
    and the whole way back run on the kernels of csrc/blocktrain.cu.  The result is contiguous [B, C, n_out], as the modules leave it, or with `points` what the
    next block's convolution reads, channels last [B, n_out, C]."""

    @staticmethod
    def forward(ctx, x, weight, gamma, beta, block, points):
        conv, norm = block.conv, block.norm                 # (gamma and beta are the norm's)
        ctx.block, ctx.pool, ctx.points = block, None if block.pool is None else block.pool._plan, points
        relu = block.activation is not None
        xp = ops.input_points(x, conv.plan)
        y = conv.plan.forward(xp, conv.packed_weight(), None, out_dtype=torch.float32, batch=x.shape[0])
        mean, rstd, out, arg = ops.block_forward(y, norm, relu, ctx.pool)
        ctx.save_for_backward(xp if ctx.needs_input_grad[1] else None, weight, gamma, y, mean, rstd, out if relu and ctx.pool is None else None, arg)
        return out if points else ops.points_to_channels(out)      # (no view: of one made in here the caller could not change a value in place)

    @staticmethod
    def backward(ctx, gy):
        xp, weight, gamma, y, mean, rstd, act, arg = ctx.saved_tensors
        conv = ctx.block.conv
        g = gy.to(torch.float32)
        if ctx.points:
            g = _aligned(g.contiguous())
        else:
            g = ops.points_to_channels(g) if g.is_contiguous() else _aligned(g.permute(0, 2, 1).contiguous())
        dy, dgamma, dbeta = ops.norm_block_backward(y, mean, rstd, gamma, act, g, ctx.pool, arg)
        need = ctx.needs_input_grad
        gx = conv.grad_plans.input_grad(dy, weight).permute(0, 2, 1).to(torch.float32) if need[0] else None
        gw = conv.grad_plans.weight_grad(dy, xp, conv.plan, weight.dtype) if need[1] else None
        return gx, gw, dgamma if need[2] else None, dbeta if need[3] else None, None, None


def block_autograd(block, x, points=False):
    """The block's training step in one function; the caller has seen to it that the block is of that form.  -> contiguous [B, C, n_out], or with `points` a
    channels-last view, for a next block that takes it as it is (ops.input_points)."""
    y = _BlockFunction.apply(x, block.conv.weight, block.norm.weight, block.norm.bias, block, points)
    return y.permute(0, 2, 1) if points else y


def knnconv_points_autograd(layer, x, relu, below=None, above=None):
    return _KnnConvPointsFunction.apply(x, layer.weight, layer.bias, layer, relu, below, above)


def knnconv_autograd(layer, x):
    """layer(x) with gradients: forward on the layer's kernels, backward as described in this module."""
    return _KnnConvFunction.apply(x, layer.weight, layer.bias, layer)
