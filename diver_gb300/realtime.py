"""Real-time path: serialized model, reference-compatible operators, frame loop.

  convert(state_dict, alpha_map)   the reference's convert.py (:17-161): sparse
                                   feature table of the 8 corners of every
                                   occupied voxel, folded/packed decoder params
  RealtimeModel.from_serialized    eval_rt.py:52-82: voxel index map, occupancy
                                   mask, three max-pooled octree levels; the
                                   packed weights re-laid out for the kernel
  RealtimeModel.render_frame       eval_rt.py:115-122: aabb_intersect, then
                                   rounds of ray_march + mlp_eval until every
                                   pixel is finished; rgb = rgba.rgb + T

The decoder kind is taken from the decoder's own layers (mlp1.4 present means
DIVeR32).  The reference chooses by feature width (convert.py:63), which sends
a DIVeR64 decoder over 32-channel features into the DIVeR32 branch and fails;
here DIVeR64 over 32 channels packs to the layout its kernel reads
(utils/mlp_evaluation64/src/mlp_eval.cu: 8288 floats).
"""
from __future__ import annotations

import math

import torch

from . import _native as N
from .decoder import Decoder, pack_realtime, premultiply_features
from .ray_march import _u8, aabb_intersect, build_octree_levels, ray_march


def convert(state_dict: dict, alpha_map: torch.Tensor, thresh: float = 1e-2) -> dict:
    """Serialized real-time model {'f','i','m','p'} from a training state dict
    (keys as DIVeR's: voxels, mlp1.*, mlp2.*) and the alpha map of prune.py."""
    sd = {k.replace("model.", ""): v for k, v in state_dict.items() if "mlp_voxel" not in k}
    voxel_mask = alpha_map > thresh
    kind = "diver32" if "mlp1.4.weight" in sd else "diver64"
    dec = Decoder.from_state_dict(kind, sd)
    voxels = sd["voxels"].float()
    dev = voxels.device
    voxel_mask = voxel_mask.to(dev)
    nv = voxels.shape[0]
    occ = torch.nonzero(voxel_mask)  # [K,3] (z, y, x) of occupied voxels
    offs = torch.stack(torch.meshgrid(*[torch.arange(2, device=dev)] * 3, indexing="ij"), -1).reshape(-1, 3)
    idx = (occ[None] + offs[:, None]).reshape(-1, 3).unique(dim=0)  # sorted lexicographically
    feats = voxels[idx[:, 0], idx[:, 1], idx[:, 2]]
    feats = premultiply_features(dec, feats) if kind == "diver32" else feats.contiguous()
    n = nv - 1
    valid = (idx < n).all(1)
    m = torch.zeros(idx.shape[0], dtype=torch.bool, device=dev)
    iv = idx[valid]
    m[valid] = voxel_mask[iv[:, 0], iv[:, 1], iv[:, 2]]
    inds = idx[:, 0] * nv * nv + idx[:, 1] * nv + idx[:, 2]
    return {"f": feats.contiguous(), "i": inds.int(), "m": m, "p": pack_realtime(dec), "kind": kind}


class RealtimeModel:
    """A resident real-time model: feature table, index map, occupancy, octree
    levels and packed decoder weights, all on one device (several can coexist)."""

    def __init__(self, features, voxel_map, voxel_masks, octrees, packed, width, voxel_num, xyzmin, voxel_size):
        self.features, self.voxel_map, self.voxel_masks = features, voxel_map, voxel_masks
        self.octrees, self.packed, self.width = octrees, packed, width
        self.voxel_num, self.xyzmin, self.voxel_size = voxel_num, xyzmin, voxel_size

    @staticmethod
    def pack_params(ref_params: torch.Tensor, width: int, device) -> torch.Tensor:
        p = ref_params.to(device=device, dtype=torch.float32).contiguous()
        out = torch.empty(N.lib().dv_realtime_packed_size(width), device=device)
        N.call("dv_realtime_pack", width, N.ptr(p), N.ptr(out), N.stream(device))
        return out

    @staticmethod
    def from_serialized(ser: dict, voxel_num: int, xyzmin: float, voxel_size: float, device="cuda",
                        width: int | None = None) -> "RealtimeModel":
        nv = voxel_num + 1
        inds = ser["i"].to(device).long()
        ii, rem = inds // (nv * nv), inds % (nv * nv)
        jj, kk = rem // nv, rem % nv
        masks = torch.zeros(voxel_num, voxel_num, voxel_num, dtype=torch.bool, device=device)
        mm = ser["m"].to(device).bool()
        masks[ii[mm], jj[mm], kk[mm]] = True
        vmap = torch.zeros(nv, nv, nv, dtype=torch.int32, device=device)
        vmap[ii, jj, kk] = torch.arange(inds.numel(), dtype=torch.int32, device=device)
        p = ser["p"]
        if width is None:
            width = 32 if p.numel() == 3168 else 64
        masks = masks.contiguous()
        return RealtimeModel(ser["f"].to(device).float().contiguous(), vmap.contiguous(), masks,
                             build_octree_levels(masks), RealtimeModel.pack_params(p, width, device), width,
                             voxel_num, xyzmin, voxel_size)

    def tc_blob(self) -> torch.Tensor:
        """Tensor-core images of the folded layers (three BF16 terms), made once
        per model from the aligned params on the device."""
        blob, written = getattr(self, "_tc_blob", None), getattr(self, "_tc_written", None)
        dev = self.packed.device
        if blob is None:
            blob = torch.empty(N.lib().dv_realtime_tc_bytes(self.width), dtype=torch.uint8, device=dev)
            N.call("dv_realtime_tc_pack", self.width, N.ptr(self.packed), N.ptr(blob), N.stream(dev))
            self.tc_err = torch.zeros(1, dtype=torch.int32, device=dev)
            written = self._tc_written = N.LastWrite()
            written.done(dev)
            self._tc_blob = blob  # last: another thread finds the rest with it
        if written is not None:  # None: loaded, finished
            written.wait(dev)  # the images may have been made on another stream than this call's
        return blob

    def mlp_eval(self, rgba, coords, v, finish, tensor_cores: bool = False):
        """One round of the fused decoder on the recorded hits (mlp_eval.cu:32-231),
        in place on rgba / finish; tensor_cores: the tcgen05 form (dv_mlp_eval_tc)."""
        fin = finish.view(torch.uint8) if finish.dtype == torch.bool else finish
        B = v.numel() // 3
        if tensor_cores:
            blob = self.tc_blob()
            N.call("dv_mlp_eval_tc", self.width, B, N.ptr(coords), N.ptr(self.features), N.ptr(self.voxel_map),
                   self.voxel_map.shape[0], N.ptr(self.packed), N.ptr(blob), N.ptr(v), N.ptr(rgba), N.ptr(fin),
                   N.ptr(self.tc_err), N.stream(v.device))
            return
        N.call("dv_mlp_eval", self.width, B, N.ptr(coords), N.ptr(self.features), N.ptr(self.voxel_map),
               self.voxel_map.shape[0], N.ptr(self.packed), N.ptr(v), N.ptr(rgba), N.ptr(fin), N.stream(v.device))

    def render_frame(self, eye: torch.Tensor, dirs: torch.Tensor, max_rounds: int | None = None,
                     fused: bool | None = None, mode: str = "tc"):
        """rgb [B,3] of B rays from camera centre `eye` (world) with unit
        directions `dirs` [B,3] (eval_rt.py:106-122); also returns the number of
        host rounds.  mode:
          "tc"     (default) the reference's loop with the tensor-core decoder
                   (FP32-grade) over the pixels still alive: dv_realtime_begin,
                   then rounds of dv_march_live + dv_mlp_eval_live until none is
                   left; a pixel gets what aabb_intersect, ray_march and
                   dv_mlp_eval_tc give it
          "fused"  the whole frame in one launch with the FP32 decoder
                   (dv_realtime_frame)
          "loop"   the reference's loop with the FP32 decoder (dv_mlp_eval);
                   same result as "fused"
        fused=True / False select "fused" / "loop" (the earlier form of this
        argument); max_rounds caps the rounds of the loops."""
        if fused is not None:
            mode = "fused" if fused else "loop"
        if mode not in ("tc", "fused", "loop"):
            raise ValueError(f"unknown real-time frame mode {mode!r}")
        dev = dirs.device
        B = dirs.shape[0]
        v = dirs.contiguous()
        center = ((eye.float().cpu() - self.xyzmin) / self.voxel_size).to(dev).contiguous()
        if center.numel() < 3:
            raise ValueError(f"eye must hold 3 coordinates, got {tuple(eye.shape)}")
        if mode == "fused":
            if v.numel() * v.element_size() < 12 * B:  # the kernel reads three floats at v + 3 b
                raise ValueError(f"dirs must hold one (x, y, z) in FP32 per ray, [B, 3], got {tuple(v.shape)} {v.dtype}")
            rgba = torch.empty(B, 4, device=dev)
            m8 = self.voxel_masks.view(torch.uint8) if self.voxel_masks.dtype == torch.bool else self.voxel_masks
            o8 = self.octrees.view(torch.uint8) if self.octrees.dtype == torch.bool else self.octrees
            N.call("dv_realtime_frame", self.width, B, N.ptr(v), N.ptr(center), N.ptr(o8), self.voxel_num, N.ptr(m8),
                   N.ptr(self.features), N.ptr(self.voxel_map), self.voxel_map.shape[0], N.ptr(self.packed),
                   N.ptr(rgba), N.stream(dev))
            return rgba[:, :3] + rgba[:, 3:], 1
        rounds = 0
        limit = max_rounds if max_rounds is not None else 3 * self.voxel_num
        if mode == "loop":
            coords = torch.zeros(8, B, 6, device=dev)
            rgba = torch.zeros(B, 4, device=dev)
            finish = torch.zeros(B, dtype=torch.bool, device=dev)
            aabb_intersect(coords, v, center, finish, rgba, self.octrees, self.voxel_num)
            while rounds < limit and not bool(finish.all()):
                ray_march(coords, v, self.voxel_masks, finish, self.voxel_num)
                self.mlp_eval(rgba, coords, v, finish, False)
                rounds += 1
            return rgba[:, :3] + rgba[:, 3:], rounds
        # "tc": every round goes over the pixels still alive, a list that the
        # previous round made on the device.  The host learns one round late that
        # it is empty, so round k + 1 is queued while it waits for round k's count
        # (a round over an empty list changes nothing; the frame is the same, the
        # round count at most one higher)
        n = self.voxel_num
        if v.shape[-1] != 3 or v.numel() != 3 * B:  # the kernels read (x, y, z) at v + 3 b
            raise ValueError(f"dirs must hold one (x, y, z) per ray, [B, 3], got {tuple(v.shape)}")
        N.need_cuda("dirs", v, torch.float32)
        N.need_cuda("center", center, torch.float32)
        m8, o8 = _u8("mask", self.voxel_masks), _u8("octrees", self.octrees)
        if n % 64 != 0 or o8.numel() != (n // 64) ** 3 + (n // 16) ** 3 + (n // 4) ** 3 or m8.numel() != n ** 3:
            raise ValueError(f"voxel_num {n} must be a multiple of 64, with {n}^3 mask cells and their octree levels")
        rgba = torch.empty(B, 4, device=dev)
        if B == 0:
            return rgba[:, :3] + rgba[:, 3:], 0
        limit = max(0, math.ceil(min(limit, 3 * n + 4)))  # a round takes at least one grid plane per live pixel
        hits = torch.empty(8, B, 6, device=dev)
        resume = torch.empty(B, 3, device=dev)
        lists = torch.empty(2, B, dtype=torch.int32, device=dev)
        counts = torch.zeros(limit + 1, dtype=torch.int32, device=dev)
        blob = self.tc_blob()
        st = N.stream(dev)
        N.call("dv_realtime_begin", B, N.ptr(v), N.ptr(center), N.ptr(o8), n, N.ptr(resume), N.ptr(rgba),
               N.ptr(lists[0]), N.ptr(counts), st)
        # of this call alone: its last round's copy is still under way when it returns, and another
        # frame of the model, on another stream or thread, waits for its own (torch's pinned pool
        # holds a freed buffer back until the copies into it have run)
        left, events = torch.zeros(2, dtype=torch.int32, pin_memory=True), (torch.cuda.Event(), torch.cuda.Event())
        while rounds < limit:
            live, after = lists[rounds % 2], lists[1 - rounds % 2]
            count = counts.data_ptr() + 4 * rounds
            N.call("dv_march_live", B, N.ptr(live), count, N.ptr(hits), N.ptr(resume), N.ptr(v), N.ptr(m8),
                   n, st)
            N.call("dv_mlp_eval_live", self.width, B, N.ptr(live), count, N.ptr(hits), N.ptr(self.features),
                   N.ptr(self.voxel_map), self.voxel_map.shape[0], N.ptr(self.packed), N.ptr(blob), N.ptr(v),
                   N.ptr(rgba), N.ptr(after), count + 4, N.ptr(self.tc_err), st)
            rounds += 1
            slot = rounds % 2
            left[slot:slot + 1].copy_(counts[rounds:rounds + 1], non_blocking=True)
            events[slot].record()
            if rounds >= 2:
                events[1 - slot].synchronize()
                if int(left[1 - slot]) == 0:
                    break
        return rgba[:, :3] + rgba[:, 3:], rounds


# --- module-level drop-in for utils.mlp_evaluation / utils.mlp_evaluation64 ------

_CURRENT: dict[int, tuple] = {}


def upload_weight(device_id: int, params: torch.Tensor, voxel_map: torch.Tensor, width: int = 32):
    """Reference upload_weight (utils/mlp_evaluation/__init__.py:30-41): makes
    (params, voxel_map) the model that `mlp_eval` uses.  The buffers stay
    per-width device tensors instead of a global texture and constant bank."""
    dev = torch.device("cuda", device_id)
    packed = RealtimeModel.pack_params(params, width, dev)
    _CURRENT[width] = (packed, voxel_map.to(dev, torch.int32).contiguous())
    return torch.Tensor([0])


def mlp_eval(rgba, coord, voxels, v, mask, width: int = 32):
    """Reference mlp_eval (utils/mlp_evaluation/__init__.py:18-28), in place on rgba / mask."""
    if width not in _CURRENT:
        raise RuntimeError("upload_weight must be called before mlp_eval")
    packed, vmap = _CURRENT[width]
    N.need_cuda("voxels", voxels, torch.float32)
    fin = mask.view(torch.uint8) if mask.dtype == torch.bool else mask
    B = v.numel() // 3
    N.call("dv_mlp_eval", width, B, N.ptr(coord), N.ptr(voxels), N.ptr(vmap), vmap.shape[0], N.ptr(packed), N.ptr(v),
           N.ptr(rgba), N.ptr(fin), N.stream(v.device))
    return torch.Tensor([0])
