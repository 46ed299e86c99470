"""Bound propagation with the dim_in axis sharded over the ranks of a process group.

Every rank holds a contiguous slice of the dim_in rows of lw/uw; lb/ub and all per-column scalars
are replicated and computed redundantly.  Linear operators (conv, matmul) need no communication:
dim_in rows are independent GEMM / conv rows.  Each nonlinearity needs the dual norm of a column
over the *whole* dim_in axis: the local unfinished accumulation is all-reduced (SUM for p = inf and
p = 2, MAX for p = 1) before the relaxation is applied to the local rows.  The sum order of the
norm changes with the number of ranks, so results agree with the single-rank run within the
per-operator tolerance, not bit for bit.

With a `faith_b200.comm.Comm` the three steps of a sharded relaxation (partial norms, all-reduce, apply) are one C
call that enqueues everything on the current stream (fb_relax_sharded_f32), the all-reduce being NCCL's or the
library's one-shot exchange over NVLink.  Without one (CPU tests of the host logic over gloo, single rank) the
partial norms are reduced through torch.distributed.  One perturbed word only: the whole dim_in axis is one norm
block here (the CNN of the benchmark perturbs every pixel), and the C entry points reject anything else.
"""
import ctypes

import torch

from . import _lib, ops
from ._lib import FB_RELU, check, load


def shard_bounds(lw, uw, rank, world, dim=-2):
    """Contiguous dim_in slice of rank `rank` (the remainder goes to the last ranks one row each)."""
    n = lw.shape[dim]
    base, rem = divmod(n, world)
    start = rank * base + max(0, rank - (world - rem))
    size = base + (1 if rank >= world - rem else 0)
    return lw.narrow(dim, start, size).contiguous(), uw.narrow(dim, start, size).contiguous()


def reduce_partials(part_l, part_u, p, group=None):
    """All-reduce of the unfinished norms over the dim_in shards (one message for both sides)."""
    import torch.distributed as dist
    if group is None and not (dist.is_available() and dist.is_initialized()):
        return part_l, part_u
    if dist.get_world_size(group) == 1:
        return part_l, part_u
    buf = torch.stack((part_l, part_u))
    dist.all_reduce(buf, op=dist.ReduceOp.MAX if p == 1 else dist.ReduceOp.SUM, group=group)
    return buf[0], buf[1]


def relax_sharded(op, lw, uw, lb, ub, p, eps, group=None, comm=None, algo=0, part_ws=None, world=None):
    """Fused concretise + relax + rescale of the local dim_in rows: partial norms, all-reduce, apply.
    comm: a faith_b200.comm.Comm -> one C call, nothing in between touches the host.
    world == 1 says that the rows are not sharded at all (no reduction, whatever process group may exist)."""
    if comm is None:
        part_l, part_u = ops.norm_partials(lw, uw, p)
        norm_l, norm_u = (part_l, part_u) if world == 1 else reduce_partials(part_l, part_u, p, group)
        return ops.relax_with_norms(op, lw, uw, lb, ub, norm_l.contiguous(), norm_u.contiguous(), p, eps)
    dev = ops._chk(lw, uw, lb, ub)
    rows, Di, Do = lb.numel() // lb.shape[-1], lw.shape[-2], lw.shape[-1]
    if part_ws is None or part_ws.numel() < 2 * rows * Do:
        part_ws = torch.empty(2 * rows * Do, device=dev)
    out = (torch.empty_like(lw), torch.empty_like(uw), torch.empty_like(lb), torch.empty_like(ub))
    with torch.cuda.device(dev):
        check(load().fb_relax_sharded_f32(comm._h, algo, op, lw.data_ptr(), uw.data_ptr(), lb.data_ptr(), ub.data_ptr(),
                                          out[0].data_ptr(), out[1].data_ptr(), out[2].data_ptr(), out[3].data_ptr(),
                                          part_ws.data_ptr(), rows, Di, Do, 1, ops.norm_code(p), float(eps), None,
                                          ops._stream()), "fb_relax_sharded_f32")
    return out


def concretize_sharded(lw, uw, lb, ub, p, eps, comm, algo=0, part_ws=None):
    """Concretisation of a dim_in shard through the communicator (fb_concretize_sharded_f32)."""
    dev = ops._chk(lw, uw, lb, ub)
    rows, Di, Do = lb.numel() // lb.shape[-1], lw.shape[-2], lw.shape[-1]
    if part_ws is None or part_ws.numel() < 2 * rows * Do:
        part_ws = torch.empty(2 * rows * Do, device=dev)
    l, u = torch.empty_like(lb), torch.empty_like(ub)
    with torch.cuda.device(dev):
        check(load().fb_concretize_sharded_f32(comm._h if comm is not None else None, algo, lw.data_ptr(), uw.data_ptr(),
                                               lb.data_ptr(), ub.data_ptr(), l.data_ptr(), u.data_ptr(), part_ws.data_ptr(),
                                               rows, Di, Do, 1, ops.norm_code(p), float(eps), ops._stream()),
              "fb_concretize_sharded_f32")
    return l, u


def conv_identity_relax(op, image_lb, image_ub, weight, bias, rows, row_start, stride, pad, p, eps, scale=1.0):
    """First convolution of an all-pixels-perturbed image and the relaxation after it (op None: convolution only), for
    the dim_in rows [row_start, row_start + rows): fb_conv2d_identity_relax_f32."""
    dev = ops._chk(image_lb, image_ub, weight, bias)
    C, H, W = image_lb.shape[-3:]
    Co, _, Kh, Kw = weight.shape
    Ho, Wo = (H + 2 * pad - Kh) // stride + 1, (W + 2 * pad - Kw) // stride + 1
    y_lw = torch.empty(1, rows, Co, Ho, Wo, device=dev)
    y_uw = torch.empty_like(y_lw)
    y_lb = torch.empty(1, Co, Ho, Wo, device=dev)
    y_ub = torch.empty_like(y_lb)
    ws = torch.empty(2 * Co * Ho * Wo, device=dev)
    with torch.cuda.device(dev):
        check(load().fb_conv2d_identity_relax_f32(-1 if op is None else op, image_lb.data_ptr(), image_ub.data_ptr(),
                                                  weight.data_ptr(), bias.data_ptr() if bias is not None else None,
                                                  float(scale), y_lw.data_ptr(), y_uw.data_ptr(), y_lb.data_ptr(),
                                                  y_ub.data_ptr(), ws.data_ptr(), rows, row_start, C, H, W, Co, Kh, Kw,
                                                  stride, pad, ops.norm_code(p), float(eps), None, ops._stream()),
              "fb_conv2d_identity_relax_f32")
    return y_lw, y_uw, y_lb, y_ub


def conv_windowed(x, weight, bias, stride, pad, row_start, H0, W0, chain):
    """A later convolution of rows that are zero outside the window their pixel reaches through `chain`, the list of
    (kernel height, kernel width, stride, padding) of the convolutions so far: the weight part through
    fb_conv2d_windowed_f32, the bias part through the ordinary kernel."""
    lw, uw, lb, ub = x
    dev = ops._chk(lw, uw, lb, ub, weight, bias)
    _, rows, C, H, W = lw.shape
    Co, _, Kh, Kw = weight.shape
    Ho, Wo = (H + 2 * pad - Kh) // stride + 1, (W + 2 * pad - Kw) // stride + 1
    y_lw = torch.empty(1, rows, Co, Ho, Wo, device=dev)
    y_uw = torch.empty_like(y_lw)
    y_lb = torch.empty(1, Co, Ho, Wo, device=dev)
    y_ub = torch.empty_like(y_lb)
    lib = load()
    flat = [int(v) for c in chain for v in c]
    chain_arr = (ctypes.c_int * max(1, len(flat)))(*flat)
    with torch.cuda.device(dev):
        check(lib.fb_conv2d_windowed_f32(lw.data_ptr(), uw.data_ptr(), weight.data_ptr(), y_lw.data_ptr(), y_uw.data_ptr(),
                                         rows, row_start, H0, W0, chain_arr, len(chain), C, H, W, Co, Kh, Kw,
                                         stride, pad, ops._stream()), "fb_conv2d_windowed_f32")
        check(lib.fb_conv2d_f32(lw.data_ptr(), uw.data_ptr(), lb.data_ptr(), ub.data_ptr(), weight.data_ptr(),
                                bias.data_ptr() if bias is not None else None, y_lw.data_ptr(), y_uw.data_ptr(),
                                y_lb.data_ptr(), y_ub.data_ptr(), 1, 0, C, H, W, Co, Kh, Kw, stride, pad, ops._stream()),
              "fb_conv2d_f32")
    return y_lw, y_uw, y_lb, y_ub


def _chain_arr(chain):
    flat = [int(v) for c in chain for v in c]
    return (ctypes.c_int * max(1, len(flat)))(*flat)


def cw_extent(H0, W0, chain):
    """Largest window (wh, ww) any pixel of an H0 x W0 image reaches through `chain`: the trailing dimensions of a compact
    tensor (fb_cw_extent)."""
    wh, ww = ctypes.c_int(0), ctypes.c_int(0)
    check(load().fb_cw_extent(H0, W0, _chain_arr(chain), len(chain), ctypes.byref(wh), ctypes.byref(ww)), "fb_cw_extent")
    return wh.value, ww.value


def cw_identity_relax(op, image_lb, image_ub, weight, bias, rows, row_start, stride, pad, p, eps, scale=1.0):
    """conv_identity_relax with compact rows: z_lw, z_uw [rows, Cout, wh, ww] (fb_cw_identity_relax_f32)."""
    dev = ops._chk(image_lb, image_ub, weight, bias)
    C, H, W = image_lb.shape[-3:]
    Co, _, Kh, Kw = weight.shape
    Ho, Wo = (H + 2 * pad - Kh) // stride + 1, (W + 2 * pad - Kw) // stride + 1
    wh, ww = cw_extent(H, W, [(Kh, Kw, stride, pad)])
    z_lw = torch.empty(rows, Co, wh, ww, device=dev)
    z_uw = torch.empty_like(z_lw)
    y_lb = torch.empty(1, Co, Ho, Wo, device=dev)
    y_ub = torch.empty_like(y_lb)
    ws = torch.empty(2 * Co * Ho * Wo, device=dev)
    with torch.cuda.device(dev):
        check(load().fb_cw_identity_relax_f32(-1 if op is None else op, image_lb.data_ptr(), image_ub.data_ptr(),
                                              weight.data_ptr(), bias.data_ptr() if bias is not None else None, float(scale),
                                              z_lw.data_ptr(), z_uw.data_ptr(), y_lb.data_ptr(), y_ub.data_ptr(), ws.data_ptr(),
                                              rows, row_start, C, H, W, Co, Kh, Kw, stride, pad, ops.norm_code(p), float(eps),
                                              None, ops._stream()), "fb_cw_identity_relax_f32")
    return z_lw, z_uw, y_lb, y_ub


def cw_conv(z_lw, z_uw, weight, stride, pad, row_start, H0, W0, chain, H, W):
    """Weight part of a later convolution on compact rows (fb_cw_conv2d_f32); `chain` leads to the input [Cin, H, W]."""
    dev = ops._chk(z_lw, z_uw, weight)
    rows, C = z_lw.shape[:2]
    Co, _, Kh, Kw = weight.shape
    wh, ww = cw_extent(H0, W0, list(chain) + [(Kh, Kw, stride, pad)])
    y_lw = torch.empty(rows, Co, wh, ww, device=dev)
    y_uw = torch.empty_like(y_lw)
    with torch.cuda.device(dev):
        check(load().fb_cw_conv2d_f32(z_lw.data_ptr(), z_uw.data_ptr(), weight.data_ptr(), y_lw.data_ptr(), y_uw.data_ptr(), rows,
                                      row_start, H0, W0, _chain_arr(chain), len(chain), C, H, W, Co, Kh, Kw, stride, pad,
                                      ops._stream()), "fb_cw_conv2d_f32")
    return y_lw, y_uw


def cw_norm_partials(z_lw, z_uw, row_start, Cin0, H0, W0, chain, H, W, p):
    """Unfinished dual-norm accumulation of every dense column over the rows of a compact tensor (fb_cw_norm_partials_f32)."""
    dev = ops._chk(z_lw, z_uw)
    rows, C = z_lw.shape[:2]
    part_l = torch.empty(C * H * W, device=dev)
    part_u = torch.empty_like(part_l)
    with torch.cuda.device(dev):
        check(load().fb_cw_norm_partials_f32(z_lw.data_ptr(), z_uw.data_ptr(), part_l.data_ptr(), part_u.data_ptr(), rows,
                                             row_start, Cin0, H0, W0, _chain_arr(chain), len(chain), C, H, W, ops.norm_code(p),
                                             ops._stream()), "fb_cw_norm_partials_f32")
    return part_l, part_u


def cw_relax_apply(op, z_lw, z_uw, lb, ub, norm_l, norm_u, row_start, H0, W0, chain, H, W, p, eps):
    """Relaxation of compact rows from given (reduced) norm accumulations (fb_cw_relax_apply_f32)."""
    dev = ops._chk(z_lw, z_uw, lb, ub, norm_l, norm_u)
    rows, C = z_lw.shape[:2]
    o_lw, o_uw, o_lb, o_ub = torch.empty_like(z_lw), torch.empty_like(z_uw), torch.empty_like(lb), torch.empty_like(ub)
    coef = torch.empty(4 * C * H * W, device=dev)
    with torch.cuda.device(dev):
        check(load().fb_cw_relax_apply_f32(op, z_lw.data_ptr(), z_uw.data_ptr(), lb.data_ptr(), ub.data_ptr(), norm_l.data_ptr(),
                                           norm_u.data_ptr(), o_lw.data_ptr(), o_uw.data_ptr(), o_lb.data_ptr(), o_ub.data_ptr(),
                                           coef.data_ptr(), rows, row_start, H0, W0, _chain_arr(chain), len(chain), C, H, W,
                                           ops.norm_code(p), float(eps), None, ops._stream()), "fb_cw_relax_apply_f32")
    return o_lw, o_uw, o_lb, o_ub


def cw_linear(z_lw, z_uw, weight, row_start, H0, W0, chain, H, W):
    """Weight rows of the linear layer that ends the spatial part, from compact rows: [rows, N] (fb_cw_linear_f32)."""
    dev = ops._chk(z_lw, z_uw, weight)
    rows, C = z_lw.shape[:2]
    N = weight.shape[0]
    y_lw = torch.empty(rows, N, device=dev)
    y_uw = torch.empty_like(y_lw)
    with torch.cuda.device(dev):
        check(load().fb_cw_linear_f32(z_lw.data_ptr(), z_uw.data_ptr(), weight.data_ptr(), y_lw.data_ptr(), y_uw.data_ptr(),
                                      y_lw.data_ptr(), rows,   # (the scratch argument is not used)
                                      row_start, H0, W0, _chain_arr(chain), len(chain), C, H, W, N, ops._stream()),
              "fb_cw_linear_f32")
    return y_lw, y_uw


def cw_expand(z_lw, z_uw, row_start, H0, W0, chain, H, W):
    """Dense rows [rows, C, H, W] of a compact tensor (fb_cw_expand_f32)."""
    dev = ops._chk(z_lw, z_uw)
    rows, C = z_lw.shape[:2]
    y_lw = torch.empty(rows, C, H, W, device=dev)
    y_uw = torch.empty_like(y_lw)
    with torch.cuda.device(dev):
        check(load().fb_cw_expand_f32(z_lw.data_ptr(), z_uw.data_ptr(), y_lw.data_ptr(), y_uw.data_ptr(), rows, row_start, H0, W0,
                                      _chain_arr(chain), len(chain), C, H, W, ops._stream()), "fb_cw_expand_f32")
    return y_lw, y_uw


class CnnVerifier:
    """Forward bound pass of conv -> relu -> conv -> relu -> linear on one image with every pixel
    perturbed (dim_in = C*H*W), the dim_in axis sharded over the ranks of `group`.

    layers: list of ("conv", weight [Co,Ci,k,k], bias, stride, pad) / ("relu",) / ("linear", W, b).
    Returns the concretised output bounds (l, u), identical on every rank.

    A network that starts with a convolution goes through the C driver (fb_cnn_forward_f32): one call enqueues the
    whole pass, the structure of the identity input is used (first convolution and its relaxation written from the
    filter alone, later convolutions windowed).  `forward(dense=True)`, and networks that start otherwise, take the
    general kernels operator by operator with the identity materialised.

    `graph` is accepted and has no effect.  Single-GPU passes used to be replayed from a CUDA graph captured per shape, norm
    and radius, which were never given up.  With five launches a pass the copies around a replay cost more than enqueueing it
    (3 x 32 x 32 image: 49.6 us a pass replayed, 44.1 us enqueued; one pass alone 60.7 and 56.1 us), and the first pass at a
    radius was a capture and an instantiation (0.8 ms and more; 57 us now).
    """

    def __init__(self, layers, device, group=None, comm=None, algo=0, compact=True, graph=True):
        self.device = torch.device(device)
        self.graph = graph      # without effect (see the class)
        self._plan = None
        self.compact = compact  # rows kept as their windows only (fb_cw_*), or dense rows (fb_conv2d_windowed_f32)
        self.group = group
        self.comm = comm        # faith_b200.comm.Comm: the all-reduces are enqueued by the library (NCCL or one-shot)
        self.algo = algo
        self._ws = None
        self._arena = None
        self.layers = []
        for ly in layers:
            if ly[0] in ("conv", "linear"):
                self.layers.append((ly[0],) + tuple(t.to(self.device, torch.float32).contiguous()
                                                    if isinstance(t, torch.Tensor) else t for t in ly[1:]))
            else:
                self.layers.append(ly)
        # the network as the C driver takes it (host array of layer records; the tensors above keep the weights alive)
        recs = (_lib.CnnLayer * max(1, len(self.layers)))()
        for r, ly in zip(recs, self.layers):
            if ly[0] == "conv":
                r.kind, r.weight, r.bias = _lib.FB_CNN_CONV, ly[1].data_ptr(), ly[2].data_ptr() if ly[2] is not None else None
                r.cout, r.kh, r.kw, r.stride, r.pad = ly[1].shape[0], ly[1].shape[2], ly[1].shape[3], ly[3], ly[4]
            elif ly[0] == "linear":
                r.kind, r.weight, r.bias = _lib.FB_CNN_LINEAR, ly[1].data_ptr(), ly[2].data_ptr() if ly[2] is not None else None
                r.n_out = ly[1].shape[0]
            else:
                r.kind = _lib.FB_CNN_RELU
        self._recs = recs
        self._driver_ok = bool(self.layers) and self.layers[0][0] == "conv"

    def _plan_for(self, C, H, W, size):
        """The network as the C driver takes it for a C x H x W image and the features of its last layer, with the arena for
        `size` rows of dim_in at hand; kept for the shape of the last call."""
        key = (C, H, W, size)
        if self._plan is None or self._plan[0] != key:
            net = _lib.Cnn(len(self.layers), self._recs, C, H, W)
            need = load().fb_cnn_workspace_bytes(ctypes.byref(net), size)
            if need < 0:
                raise _lib.FaithError("fb_cnn_workspace_bytes: network not supported by the driver")
            if self._arena is None or self._arena.numel() < need:
                self._arena = torch.empty(need, dtype=torch.uint8, device=self.device)
            self._plan = (key, net, self._out_features(C, H, W))
        return self._plan

    def _forward_driver(self, image, p, eps, start, size, world):
        """One fb_cnn_forward_f32 call on the current stream."""
        _, net, n_out = self._plan_for(*image.shape, size)
        img = image.to(self.device, torch.float32, non_blocking=True).contiguous()
        comm = self.comm._h.value if (self.comm is not None and world > 1) else None
        out = _lib.binding().cnn_forward(ctypes.addressof(net), img, p, eps, start, size, comm, self.algo, 1 if self.compact else 0,
                                         n_out, self._arena)
        return out.unbind(0)

    def _out_features(self, C, H, W):
        c, h, w = C, H, W
        feat = c * h * w
        for ly in self.layers:
            if ly[0] == "conv":
                k_h, k_w = ly[1].shape[2], ly[1].shape[3]
                h, w, c = (h + 2 * ly[4] - k_h) // ly[3] + 1, (w + 2 * ly[4] - k_w) // ly[3] + 1, ly[1].shape[0]
                feat = c * h * w
            elif ly[0] == "linear":
                feat = ly[1].shape[0]
        return feat

    def forward(self, image, p, eps, rank=0, world=1, dense=False):
        """dense=True materialises the identity input and runs every convolution densely, operator by operator (the
        general kernels; kept for comparison).  Otherwise the C driver runs the pass."""
        C, H, W = image.shape
        di = C * H * W
        base, rem = divmod(di, world)
        start = rank * base + max(0, rank - (world - rem))
        size = base + (1 if rank >= world - rem else 0)
        if not dense and self._driver_ok and (world == 1 or self.comm is not None):
            return self._forward_driver(image, p, eps, start, size, world)
        lb = image.to(self.device, torch.float32).view(1, C, H, W).contiguous()
        ub = lb.clone()
        layers = list(self.layers)
        chain = None      # geometry of the convolutions so far, while the rows keep their window structure
        if dense or not layers or layers[0][0] != "conv":
            # identity dependence on every pixel: the local rows of eye(di)
            lw = torch.zeros(size, di, device=self.device)
            lw[torch.arange(size, device=self.device), start + torch.arange(size, device=self.device)] = 1.0
            lw = lw.view(1, size, C, H, W)
            uw = lw.clone()
        else:
            ly = layers.pop(0)
            fuse = bool(layers) and layers[0][0] == "relu"
            if fuse:
                layers.pop(0)
            lw, uw, lb, ub = conv_identity_relax(FB_RELU if fuse else None, lb, ub, ly[1], ly[2], size, start, ly[3], ly[4],
                                                 p, eps)
            chain = [(ly[1].shape[-2], ly[1].shape[-1], ly[3], ly[4])]
        for ly in layers:
            if ly[0] == "conv" and chain is not None:
                lw, uw, lb, ub = conv_windowed((lw, uw, lb, ub), ly[1], ly[2], ly[3], ly[4], start, H, W, chain)
                chain.append((ly[1].shape[-2], ly[1].shape[-1], ly[3], ly[4]))
            elif ly[0] == "conv":
                lw, uw, lb, ub = ops.conv2d((lw, uw, lb, ub), ly[1], ly[2], ly[3], ly[4])
            elif ly[0] == "relu":
                shp_w, shp_b = lw.shape, lb.shape
                comm = self.comm if world > 1 else None
                if comm is not None and (self._ws is None or self._ws.numel() < 2 * lb.numel()):
                    self._ws = torch.empty(2 * lb.numel(), device=self.device)
                o = relax_sharded(FB_RELU, lw.reshape(1, size, -1), uw.reshape(1, size, -1), lb.reshape(1, -1),
                                  ub.reshape(1, -1), p, eps, self.group, comm, self.algo, self._ws, world)
                lw, uw, lb, ub = o[0].view(shp_w), o[1].view(shp_w), o[2].view(shp_b), o[3].view(shp_b)
            elif ly[0] == "linear":
                lw, uw, lb, ub = ops.matmul(lw.reshape(1, 1, size, -1), uw.reshape(1, 1, size, -1),
                                            lb.reshape(1, 1, -1), ub.reshape(1, 1, -1), ly[1], ly[2])
        if self.comm is not None and world > 1:
            l, u = concretize_sharded(lw.reshape(1, size, -1), uw.reshape(1, size, -1), lb.reshape(1, -1), ub.reshape(1, -1),
                                      p, eps, self.comm, self.algo)
            return l.reshape(-1), u.reshape(-1)
        part_l, part_u = ops.norm_partials(lw.reshape(1, size, -1), uw.reshape(1, size, -1), p)
        norm_l, norm_u = (part_l, part_u) if world == 1 else reduce_partials(part_l, part_u, p, self.group)
        if p == 2:
            norm_l, norm_u = norm_l.sqrt(), norm_u.sqrt()
        return lb.reshape(-1) - eps * norm_l.reshape(-1), ub.reshape(-1) + eps * norm_u.reshape(-1)
