"""One-call form of the backbone's forward (ptv3_backbone_fwd): the argument blocks of a network
whose modules all have their standard form, kept between passes and rebuilt when a parameter, a
buffer or a setting changed.  Weights are read where the parameters are, on every pass (fp32 networks have
them split for the tensor cores by the call)."""
import ctypes
import itertools
import operator
import weakref

import torch
import torch.nn as nn

from . import _lib, ops
from . import sparse as spconv
from .sparse import SparseConvTensor

_GLOBAL_HOOKS = nn.modules.module


def _exact_gelu(m):
    return type(m) is nn.GELU and getattr(m, "approximate", "none") == "none"


def _eval_bn(m):
    return type(m) is nn.BatchNorm1d and m.track_running_stats


class _Unsupported(Exception):
    pass


def _require(ok):
    if not ok:
        raise _Unsupported


class NativeBackbone:
    """Argument blocks of ``net`` (bf16 or fp32).  ``current`` tells whether they still describe it.

    Looking a network over takes 0.14 ms of host time, half of what passes before a pass's first kernel is
    queued.  A network that stood up to it in its last pass is therefore looked over while the GPU works on
    this one: the pass is queued if everything the blocks point to is still in place (``intact``), and given
    up, unseen, if the network turns out to have changed (6 000 points: 1.77 -> 1.67 ms per pass, 100 000: 3.22 -> 3.01)."""

    def __init__(self, net):
        from . import model as M
        self.trusted = False     # the last pass found the network as the blocks have it
        self.dtype = next(net.parameters()).dtype
        self.f32 = self.dtype == torch.float32
        _require(self.dtype in (torch.float32, torch.bfloat16))
        self.refs = []           # (owner dict, name): every tensor the blocks point to
        self.norms = []          # BatchNorm and LayerNorm layers
        self.keep = []           # arrays the blocks point into
        self.modules = [m.__dict__ for m in net.modules()]
        self.parents = [d["_modules"] for d in self.modules if d["_modules"]]
        self.children = [c for d in self.parents for c in d.values()]
        _require(not net.cls_mode and len(net.order) <= 8)
        stem = list(net.embedding.stem._modules.values())
        _require(type(net.embedding) is M.Embedding and len(stem) == 3)
        conv, bn, act = stem
        _require(type(conv) is spconv.SubMConv3d and conv.uses_direct_path() and conv.bias is None
                 and _eval_bn(bn) and _exact_gelu(act))
        a = self.args = _lib.BackboneArgs()
        a.dtype, a.plain_weights = _lib.DTYPE_IDS[self.dtype], 1
        a.stem_c_in, a.stem_c_out, a.stem_ksize = conv.in_channels, conv.out_channels, conv.kernel_size
        a.stem_weight = self._param(conv, "weight")
        a.stem_bn = self._bn(bn)
        self.width_in = conv.in_channels
        enc, dec = list(net.enc._modules.values()), list(net.dec._modules.values())
        _require(len(enc) == net.num_stages and len(dec) == net.num_stages - 1 and len(enc) >= 2)
        self.blocks, self.pools = [], []
        a.n_enc, a.n_dec, a.k = len(enc), len(dec), len(net.order)
        a.enc, a.dec = self._stages(enc, True), self._stages(dec, False)
        self.width_out = self.blocks[-1].channels
        _require(self.stage_blocks[-1] >= 1)
        self.settings = self._settings()
        self.owners, self.names = [d for d, _ in self.refs], [k for _, k in self.refs]
        self.tensors = [d[k] for d, k in self.refs]
        self.ptrs = [t.data_ptr() for t in self.tensors]

    # -- what the blocks are made of
    def _param(self, module, name):
        t = module._parameters[name]
        _require(t is not None and t.dtype == self.dtype and t.is_cuda and t.is_contiguous())
        self.refs.append((module._parameters, name))
        return t.data_ptr()

    def _bn(self, bn):
        got = ops.bn_args(bn) if _eval_bn(bn) else None
        _require(got is not None)
        args, refs = got
        self.refs.extend(refs)
        self.norms.append(bn)
        self.keep.append(args)
        return ctypes.addressof(args)

    def _linear(self, lin, supported):
        _require(type(lin) is nn.Linear and lin.bias is not None
                 and (lin.in_features % 32 == 0 and lin.out_features % 32 == 0 if self.f32
                      else supported(lin.in_features, lin.out_features, torch.bfloat16)))
        return self._param(lin, "weight"), self._param(lin, "bias")

    def _stages(self, stages, encoder):
        from . import model as M
        out = (_lib.StageArgs * len(stages))()
        self.stage_blocks = []
        for s, (stage, st) in enumerate(zip(stages, out)):
            mods = list(stage._modules.values())
            if not encoder:
                up = mods.pop(0)
                _require(type(up) is M.SerializedUnpooling and not up.traceable and up._fusable_form())
                st.c_in, st.c_skip = up.proj[0].in_features, up.proj_skip[0].in_features
                st.c_out = up.proj[0].out_features
                _require(up.proj_skip[0].out_features == st.c_out)
                st.w, st.b = self._linear(up.proj[0], ops.pool_stage_supported)
                st.w_skip, st.b_skip = self._linear(up.proj_skip[0], ops.pool_stage_supported)
                st.bn = self._bn(up.proj[1])
                st.bn_skip = self._bn(up.proj_skip[1])
            elif s > 0:
                _require(mods and type(mods[0]) is M.SerializedPooling)
                down = mods.pop(0)
                _require(down.norm is not None and down.act is not None and len(down.norm) == 1 and len(down.act) == 1
                         and _exact_gelu(down.act[0]))
                st.c_in, st.c_out = down.proj.in_features, down.proj.out_features
                st.w, st.b = self._linear(down.proj, ops.pool_stage_supported)
                st.bn = self._bn(down.norm[0])
                st.pooling_depth, st.reduce = down.pooling_depth(), ops.REDUCE_IDS[down.reduce]
                self.pools.append(down)
            blocks = (_lib.BlockArgs * max(1, len(mods)))()
            order_index, patch = (ctypes.c_int * max(1, len(mods)))(), (ctypes.c_int * max(1, len(mods)))()
            for j, m in enumerate(mods):
                _require(type(m) is M.Block and m._fusable_form() and not m.attn.enable_rpe
                         and type(m.attn) is M.SerializedAttention and m._native_static_ok(self.dtype, f32=self.f32)
                         and m.channels < spconv.PAIR_PATH_MIN_CHANNELS)
                args = m._native_args(self.dtype, m.attn.qkv.weight.device)
                _require(args is not None and args.conv_weight)
                ctypes.pointer(blocks[j])[0] = args
                self.refs.extend(m.__dict__["_ptv3_block_args"][0])
                order_index[j] = m.attn.order_index
                patch[j] = m.attn.patch_size if m.attn.enable_flash else -m.attn.patch_size_max
                self.blocks.append(m)
                self.norms.extend(m.__dict__["_ptv3_block_args"][4])
            st.n_blocks, st.blocks, st.order_index, st.patch = len(mods), blocks, order_index, patch
            self.stage_blocks.append(len(mods))
            self.keep.append((blocks, order_index, patch))
        self.keep.append(out)
        return out

    def _settings(self):
        got = []
        for m in self.blocks:
            t = m.attn
            got.append((t.algo, t.scale, t.order_index, t.enable_flash,
                        t.patch_size if t.enable_flash else t.patch_size_max))
        for p in self.pools:
            got.append((p.stride, p.reduce))
        got.extend([norm.eps for norm in self.norms])
        return got

    def current(self):
        """Whether every module, parameter, buffer and setting is as it was when the blocks were made."""
        children = list(itertools.chain.from_iterable(map(dict.values, self.parents)))
        return (len(children) == len(self.children) and all(map(operator.is_, children, self.children))
                and all(map(operator.is_, map(dict.get, self.owners, self.names), self.tensors))
                and list(map(torch.Tensor.data_ptr, self.tensors)) == self.ptrs
                and self._settings() == self.settings)

    def observed(self):
        """Whether someone looks at (or changed the mode of) single modules: the module tree is then run itself."""
        return (any(map(operator.itemgetter("training"), self.modules))
                or any(map(operator.itemgetter("_forward_hooks"), self.modules))
                or any(map(operator.itemgetter("_forward_pre_hooks"), self.modules))
                or bool(_GLOBAL_HOOKS._global_forward_hooks) or bool(_GLOBAL_HOOKS._global_forward_pre_hooks))

    def intact(self, net):
        """Whether the blocks can be run on: the memory they point to is there (and the network was neither put
        into training mode nor given another number of orders, which would make the pass one for nothing)."""
        return (not net.training and len(net.order) == self.args.k
                and list(map(torch.Tensor.data_ptr, self.tensors)) == self.ptrs)

    # -- one pass
    def run(self, net, point, depth, side, checked):
        """The forward of ``point`` (features, grid coordinates, offset, host counts and sparse shape
        in place); leaves the Point of the finest level in it.  ``checked``: the network was looked over; else
        that happens here, and None with ``point`` and the random state as they were means that it changed."""
        rng = None if checked else torch.get_rng_state()
        n, k, counts = point.feat.shape[0], len(net.order), point["_counts"]
        n_scenes = len(counts)
        order = list(net.order)
        if net.shuffle_orders:
            order = [order[i] for i in torch.randperm(k).tolist()]
        perms = None
        if self.pools:
            perms = (ctypes.c_int * (len(self.pools) * k))()
            for i, p in enumerate(self.pools):
                perms[i * k:(i + 1) * k] = torch.randperm(k).tolist() if p.shuffle_orders else range(k)
        feat, dev = point.feat.contiguous(), point.feat.device
        grid = point.grid_coord.to(torch.int32).contiguous()
        offset, batch = point.offset.to(torch.int64).contiguous(), point.batch.to(torch.int64).contiguous()
        code, sorted_order, inverse = (torch.empty((k, n), dtype=torch.int64, device=dev) for _ in range(3))
        indices = torch.empty((n, 4), dtype=torch.int32, device=dev)
        nbr = torch.empty((27, n), dtype=torch.int32, device=dev)
        out = torch.empty((n, self.width_out), dtype=feat.dtype, device=dev)
        status = point.device_status()
        pad = unpad = cu = None
        patch = 0
        if self.stage_patch0():
            patch = self.stage_patch0()
            if patch < 0:
                patch = min(min(counts), -patch)
            n_pad, n_seq = ops.pad_layout(counts, patch)
            pad = torch.empty(n_pad, dtype=torch.int64, device=dev)
            unpad = torch.empty(n, dtype=torch.int64, device=dev)
            cu = torch.empty(n_seq + 1, dtype=torch.int32, device=dev)
        a = _lib.BackboneArgs.from_buffer_copy(self.args)      # passes of several threads do not share one
        host_counts = (ctypes.c_int64 * n_scenes)(*counts)
        level_counts = (ctypes.c_int64 * (a.n_enc * n_scenes))()
        ids = (ctypes.c_int * k)(*[ops.ORDER_IDS[o] for o in order])
        main = torch.cuda.current_stream()
        meta = ops._host_words((a.n_enc - 1) * (3 + n_scenes), "backbone.meta", main.cuda_stream)
        chunks, failed = ([], []), []

        def alloc(_, nbytes, pool):
            try:
                if pool:
                    with torch.cuda.stream(side):
                        t = torch.empty(nbytes, dtype=torch.uint8, device=dev)
                else:
                    t = torch.empty(nbytes, dtype=torch.uint8, device=dev)
                chunks[pool].append(t)
                return t.data_ptr()
            except Exception as e:                             # out of memory: raised below
                failed.append(e)
                return None

        a.n, a.n_scenes, a.depth = n, n_scenes, depth
        a.counts, a.order_ids, a.row_perm = host_counts, ids, perms
        a.feat, a.grid_coord, a.offset, a.batch = feat.data_ptr(), grid.data_ptr(), offset.data_ptr(), batch.data_ptr()
        a.code, a.order, a.inverse = code.data_ptr(), sorted_order.data_ptr(), inverse.data_ptr()
        a.indices, a.nbr, a.out = indices.data_ptr(), nbr.data_ptr(), out.data_ptr()
        if pad is not None:
            a.pad, a.unpad, a.cu_seqlens = pad.data_ptr(), unpad.data_ptr(), cu.data_ptr()
        a.level_counts, a.meta_host, a.status = level_counts, meta.address, status.data_ptr()
        a.alloc = _lib.ALLOC_FN(alloc)
        a.main_stream, a.plan_stream = main.cuda_stream, side.cuda_stream
        rc = _lib.load().ptv3_backbone_fwd(ctypes.byref(a))
        self.trusted = checked or (self.current() and not self.observed())
        if rc != 0 or not self.trusted:
            message = _lib.load().ptv3_last_error().decode()
            torch.cuda.synchronize()                           # nothing queued may outlive its memory
            if not self.trusted:
                torch.set_rng_state(rng)
                return None
            if failed:
                raise failed[0]
            raise _lib.Ptv3Error("ptv3_backbone_fwd failed (%d): %s" % (rc, message))
        # planning memory belongs to the planning stream and was read on the main stream too
        for t in chunks[1]:
            t.record_stream(main)
        for i, m in enumerate(self.blocks):
            if not m.attn.enable_flash:
                s = self.level_of_block(i)
                level = level_counts[s * n_scenes:(s + 1) * n_scenes]
                m.attn.patch_size = min(min(level), m.attn.patch_size_max)
        point["serialized_depth"] = depth
        point["serialized_code"], point["serialized_order"], point["serialized_inverse"] = code, sorted_order, inverse
        if pad is not None and self.stage_patch0() == self.last_patch():
            point["pad"], point["unpad"], point["cu_seqlens_key"], point["_pad_patch"] = pad, unpad, cu, patch
        point["feat"] = out
        point["sparse_conv_feat"] = SparseConvTensor(
            features=out, indices=indices, spatial_shape=point["sparse_shape"], batch_size=n_scenes,
            row_order=sorted_order[0], status=status, defer_status=True, prebuilt={3: (nbr, sorted_order[0])})
        return point

    def stage_patch0(self):
        st = self.args.enc[0]
        return st.patch[0] if st.n_blocks else 0

    def last_patch(self):
        st = self.args.dec[self.args.n_dec - 1]
        return st.patch[st.n_blocks - 1]

    def level_of_block(self, i):
        """Resolution level of the i-th block (encoder blocks first)."""
        for s in range(self.args.n_enc):
            if i < self.args.enc[s].n_blocks:
                return s
            i -= self.args.enc[s].n_blocks
        for d in range(self.args.n_dec):
            if i < self.args.dec[d].n_blocks:
                return self.args.n_enc - 2 - d
            i -= self.args.dec[d].n_blocks
        raise IndexError(i)


_NATIVE = weakref.WeakKeyDictionary()     # network -> its NativeBackbone, or what was looked at in vain


def of(net):
    """The NativeBackbone of ``net``, or None where a module has another form than the standard one or is
    observed; and whether the network was looked over for that."""
    native = _NATIVE.get(net)
    if isinstance(native, NativeBackbone):
        if native.trusted and native.intact(net):
            return native, False
        if native.current():
            return None if native.observed() else native, True
    elif native is not None and native == _seen(net):
        return None, True
    try:
        native = _NATIVE[net] = NativeBackbone(net)
        return None if native.observed() else native, True
    except (_Unsupported, KeyError, IndexError, AttributeError):
        _NATIVE[net] = _seen(net)
        return None, True


def _seen(net):
    """Tells a network that was not taken from the same one after a conversion."""
    p = next(net.parameters())
    return p.dtype, p.device, p.data_ptr()
