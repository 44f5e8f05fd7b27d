"""GPU: the tensor-core decoder at the edges of its 128-segment tiles and of
one launch's resident tiles (past them the forward's tiles come from cluster
launch control), with the segment count held by the host or by the device; the
split backward at the edges of its tiles and of one tile per SM.  The plain
FP32 kernels are the reference.  Tolerances: forward, the forms' stated ones
(per segment 3e-2 BF16, 4e-3 FP16, 1e-5 split, of max(1, largest density));
split gradients 2e-5 relative L2: two BF16 terms leave at most 2^-18 of each
operand, 2^-17 = 8e-6 of a product, doubled for what cancels in the sums."""
import pytest
import torch

from tests.test_decode_plain_tiles_gpu import case

pytestmark = pytest.mark.gpu
TOL = {"bf16": 3e-2, "fp16": 4e-3, "bf16s": 1e-5}
SIZES = [1, 127, 128, 129, 160_001]  # the last: past one wave of 152 SMs x 8 tiles


class Lists:
    """Segment lists with the count on the host (exact) or on the device."""

    def __init__(self, seg, ray, count=None):
        self.seg, self.ray, self.total, self.count = seg, ray, seg.shape[0], count
        self.count_ptr = None if count is None else count.data_ptr()


def setup(kind, channels, n):
    from diver_gb300 import _native as N
    from diver_gb300.decoder import pack_plain

    base = min(n, 1000)  # longer lists repeat the walk
    vox, seg, ray, dirs, dec, _ = case(base, channels, kind, 3 * base + channels)
    dec.layers[dec.n_mlp1 - 1][1][0] += 0.6  # active density
    vox = vox / 6  # the stated tolerances' feature size
    reps = -(-n // base)
    B = dirs.shape[0]
    ray = torch.cat([ray + i * B for i in range(reps)])[:n]
    dv, ds, dr, dd, dp = (x.cuda().contiguous() for x in (vox, seg.repeat(reps, 1)[:n], ray, dirs.repeat(reps, 1),
                                                         pack_plain(dec)))
    pe = torch.empty(dd.shape[0], 28, device="cuda"), torch.empty(dd.shape[0], dec.width, device="cuda")
    st = N.stream(dv.device)
    N.call("dv_ray_pe", int(kind[5:]), channels, N.ptr(dp), dd.shape[0], N.ptr(dd), N.ptr(pe[0]), N.ptr(pe[1]), st)
    ref = torch.empty(n, 4, device="cuda")
    N.call("dv_decode_fwd", int(kind[5:]), channels, N.ptr(dp), N.ptr(dv), 10, 8, 6, N.ptr(ds), N.ptr(dr), n, None,
           N.ptr(pe[1]), N.ptr(ref), st)
    return dec, dv, dp, Lists(ds, dr), pe, ref, st


@pytest.mark.parametrize("kind,channels", [("diver32", 32), ("diver64", 32), ("diver64", 64)])
@pytest.mark.parametrize("form", ["bf16", "fp16", "bf16s"])
@pytest.mark.parametrize("n", SIZES)
def test_tc_forward_tile_edges(kind, channels, form, n):
    from diver_gb300.renderer import TcWeights

    dec, dv, dp, seg, pe, ref, st = setup(kind, channels, n)
    k = int(kind[5:])
    tw = TcWeights.from_decoder(dec, "cuda", mode=form)
    pad = torch.cat([seg.seg, seg.seg[:1].repeat(200, 1)]), torch.cat([seg.ray, seg.ray[:1].repeat(200)])
    device = Lists(*pad, torch.tensor([n], device="cuda"))
    for g16 in (None,) if form == "bf16s" else (None, dv.to(tw.dtype)):
        got, got2 = torch.full_like(ref, -7.0), torch.full((n + 200, 4), -7.0, device="cuda")
        tw.decode(k, channels, dv, seg, pe[1], got, st, g16)
        tw.decode(k, channels, dv, device, pe[1], got2, st, g16)
        torch.cuda.synchronize()
        assert int(tw.err.item()) == 0
        err = (got - ref).abs().max(0).values
        assert err[0] <= TOL[form] * max(1.0, float(ref[:, 0].abs().max())) and err[1:].max() <= TOL[form]
        assert torch.equal(got2[:n], got) and bool((got2[n:] == -7.0).all())


@pytest.mark.parametrize("n", [1, 127, 128, 129, 152 * 128, 152 * 128 + 1])
def test_split_backward_tile_edges(n):
    """Both forms of the split backward: mlp1's output layer and mlp2's first
    as one (TcWeights.backward) and layer by layer."""
    from diver_gb300 import _native as N
    from diver_gb300.decoder import pack_tc_bwd, tc_index_maps
    from diver_gb300.renderer import TcWeights

    dec, dv, dp, seg, pe, _, st = setup("diver32", 32, n)
    tw = TcWeights.from_decoder(dec, "cuda", mode="bf16s")
    out4 = torch.empty(n, 4, device="cuda")
    save = tw.save_buffer(32, 32, n, "cuda")
    tw.decode(32, 32, dv, seg, pe[1], out4, st, None, save)
    d4 = torch.randn(n, 4, generator=torch.Generator().manual_seed(n)).cuda()
    grid = (10, 8, 6, N.ptr(seg.seg), N.ptr(seg.ray), n, None)
    grads = [(torch.zeros_like(dv), torch.zeros_like(dp)) for _ in range(3)]
    N.call("dv_decode_bwd", 32, 32, N.ptr(dp), N.ptr(dv), *grid, N.ptr(pe[0]), N.ptr(pe[1]), N.ptr(d4),
           *(N.ptr(x) for x in grads[0]), st)
    assert tw.backward(32, dv, seg, *pe, d4, *grads[1], st, save, out4)
    maps = tc_index_maps("diver32", 32)
    index, table = maps["bwd"].cuda(), maps["bwd_table"].contiguous()
    wb = torch.empty(3 * index.numel(), dtype=torch.bfloat16, device="cuda")
    N.call("dv_tc_image", N.ptr(dp), dp.numel(), N.ptr(index), index.numel(), 3, N.ptr(wb), st)
    assert torch.equal(wb[:index.numel()].cpu(), pack_tc_bwd(dec)[0].view(torch.bfloat16).reshape(-1))
    N.call("dv_decode_fwd_tc_split", 32, 32, N.ptr(tw.blob), tw.term_bytes, N.ptr(tw.bias), tw.bias.numel(),
           tw.table.data_ptr(), tw.table.shape[0], N.ptr(dv), *grid, N.ptr(pe[1]), N.ptr(out4), N.ptr(save), save.numel(),
           N.ptr(tw.err), st)  # the record of every layer
    N.call("dv_decode_bwd_tc_split", 32, 32, N.ptr(wb), 2 * index.numel(), table.data_ptr(), table.shape[0], *grid,
           N.ptr(pe[0]), N.ptr(d4), N.ptr(save), save.numel(), N.ptr(out4), *(N.ptr(x) for x in grads[2]), None,
           N.ptr(tw.err), st)
    torch.cuda.synchronize()
    assert int(tw.err.item()) == 0
    for got in grads[1:]:
        for a, b in zip(got, grads[0]):
            assert (a - b).norm() <= 2e-5 * b.norm()
