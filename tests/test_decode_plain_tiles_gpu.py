"""GPU: the per-ray encoding at the edges of its blocks' turns, and the plain
FP32 decoder, forward and backward, at the edges of its
16- and 32-segment warp tiles and of the backward's 128-segment steps, with
rays that end inside tiles and segments on the grid's far faces, against the
FP64 oracle.  Tolerances: forward 1e-5 abs, gradients 1e-4 relative L2, the
plain form's stated ones."""
import pytest
import torch

from oracle import torch_ref

pytestmark = pytest.mark.gpu
SIZES = [1, 15, 16, 17, 31, 32, 33, 127, 128, 129, 1000]


def case(n, channels, kind, seed):
    from diver_gb300.decoder import random_decoder

    g = torch.Generator().manual_seed(seed)
    dims = torch.tensor([9, 7, 5])
    vox = torch.randn(6, 8, 10, channels, generator=g) * 0.3
    # a walk through face-adjacent cells with jumps, some cells at the far faces
    cell = (torch.rand(n, 3, generator=g) * dims).long()
    for i in range(1, n):
        if torch.rand((), generator=g) < 0.7:
            step = torch.zeros(3, dtype=torch.long)
            step[int(torch.randint(0, 3, (1,), generator=g))] = 1 if torch.rand((), generator=g) < 0.5 else -1
            cell[i] = torch.minimum((cell[i - 1] + step).clamp_min(0), dims - 1)
    p = cell[:, None, :] + 0.01 + 0.98 * torch.rand(n, 2, 3, generator=g)
    ray = torch.cumsum((torch.rand(n, generator=g) < 0.1).long(), 0)
    ray = (ray - ray[0]).int()
    dirs = torch.randn(int(ray[-1]) + 1, 3, generator=g)
    dirs = dirs / dirs.norm(dim=-1, keepdim=True)
    return vox, p.reshape(n, 6).float(), ray, dirs, random_decoder(kind, channels, seed), torch.randn(n, 4, generator=g)


@pytest.mark.parametrize("kind,channels", [("diver32", 32), ("diver64", 32), ("diver64", 64)])
@pytest.mark.parametrize("n", SIZES)
def test_plain_decoder_tile_edges(kind, channels, n):
    from diver_gb300 import _native as N
    from diver_gb300.decoder import pack_plain, unpack_plain_grad

    vox, seg, ray, dirs, dec, d4 = case(n, channels, kind, 7 * n + channels)
    k, B, W = int(kind[5:]), dirs.shape[0], dec.width
    dv, ds, dr, dd, dp, dg = (x.cuda().contiguous() for x in (vox, seg, ray, dirs, pack_plain(dec), d4))
    st = N.stream(dv.device)
    pe_feat, pe_out, out4 = (torch.empty(*s, device="cuda") for s in ((B, 28), (B, W), (n, 4)))
    gv, gp = torch.zeros_like(dv), torch.zeros_like(dp)
    grid = (N.ptr(dv), 10, 8, 6, N.ptr(ds), N.ptr(dr), n, None)
    N.call("dv_ray_pe", k, channels, N.ptr(dp), B, N.ptr(dd), N.ptr(pe_feat), N.ptr(pe_out), st)
    N.call("dv_decode_fwd", k, channels, N.ptr(dp), *grid, N.ptr(pe_out), N.ptr(out4), st)
    N.call("dv_decode_bwd", k, channels, N.ptr(dp), *grid, N.ptr(pe_feat), N.ptr(pe_out), N.ptr(dg), N.ptr(gv),
           N.ptr(gp), st)

    v64 = vox.double().requires_grad_(True)
    layers = [(w.double().requires_grad_(True), b.double().requires_grad_(True)) for w, b in dec.layers]
    feat = torch_ref.integrate(v64, seg[:, :3].double(), seg[:, 3:].double(), per_axis=True)
    sigma, rgb = torch_ref.decode(layers, dec.n_mlp1, feat, dirs.double()[ray.long()])
    ref = torch.cat([sigma[:, None], rgb], 1)
    (ref * d4.double()).sum().backward()
    assert (out4.cpu().double() - ref.detach()).abs().max() < 1e-5
    assert (gv.cpu().double() - v64.grad).norm() <= 1e-4 * v64.grad.norm()
    for (gw, gb), (w, b) in zip(unpack_plain_grad(kind, channels, gp.cpu().double()), layers):
        assert (gw - w.grad).norm() <= 1e-4 * w.grad.norm()
        assert (gb - b.grad).norm() <= 1e-4 * b.grad.norm()


@pytest.mark.parametrize("kind,channels", [("diver32", 32), ("diver64", 32), ("diver64", 64)])
@pytest.mark.parametrize("n", [1, 16, 17, 31, 32, 33, 1000, 40001])
@pytest.mark.parametrize("held", [False, True])
def test_plain_record_is_the_recompute(kind, channels, n, held):
    """The forward's record gives the recomputing backward's gradients: the
    same values in, so they differ by the order of their atomic sums only (1e-6
    relative L2).  held: the count on the device, in lists with room to spare."""
    from diver_gb300 import _native as N
    from diver_gb300.decoder import pack_plain

    base = min(n, 1000)
    vox, seg, ray, dirs, dec, _ = case(base, channels, kind, 5 * base)
    k, W = int(kind[5:]), dec.width
    rep, room, B = -(-n // base), 100 if held else 0, dirs.shape[0]
    ray = torch.cat([ray + i * B for i in range(rep)])[:n]
    seg, dirs = seg.repeat(rep, 1)[:n], dirs.repeat(rep, 1)
    seg, ray = torch.cat([seg, seg[:1].expand(room, 6)]), torch.cat([ray, ray[:1].expand(room)])
    d4 = torch.randn(n + room, 4, generator=torch.Generator().manual_seed(n))
    dv, ds, dr, dd, dp, dg = (x.cuda().contiguous() for x in (vox, seg, ray, dirs, pack_plain(dec), d4))
    count = torch.tensor([n], device="cuda") if held else None
    st, S = N.stream(dv.device), n + room
    pe_feat, pe_out = torch.empty(len(dirs), 28, device="cuda"), torch.empty(len(dirs), W, device="cuda")
    N.call("dv_ray_pe", k, channels, N.ptr(dp), len(dirs), N.ptr(dd), N.ptr(pe_feat), N.ptr(pe_out), st)
    head = (k, channels, N.ptr(dp), N.ptr(dv), 10, 8, 6, N.ptr(ds), N.ptr(dr), S, N.ptr(count))
    save = torch.empty(N.lib().dv_decode_save_bytes(k, channels, S), dtype=torch.uint8, device="cuda")
    out, out2 = torch.zeros(S, 4, device="cuda"), torch.zeros(S, 4, device="cuda")
    N.call("dv_decode_fwd", *head, N.ptr(pe_out), N.ptr(out), st)
    N.call("dv_decode_fwd_save", *head, N.ptr(pe_out), N.ptr(out2), N.ptr(save), save.numel(), st)
    assert torch.equal(out, out2)
    grads = [(torch.zeros_like(dv), torch.zeros_like(dp)) for _ in range(2)]
    tail = (N.ptr(pe_feat), N.ptr(pe_out), N.ptr(dg))
    N.call("dv_decode_bwd", *head, *tail, *(N.ptr(x) for x in grads[0]), st)
    N.call("dv_decode_bwd_saved", *head, *tail, *(N.ptr(x) for x in grads[1]), N.ptr(save), save.numel(), st)
    for a, b in zip(*grads):
        assert (a - b).norm() <= 1e-6 * b.norm()
    with pytest.raises(RuntimeError):
        N.call("dv_decode_fwd_save", *head, N.ptr(pe_out), N.ptr(out2), N.ptr(save), save.numel() - 1, st)


@pytest.mark.parametrize("kind", ["diver32", "diver64"])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 32, 33, 304 * 16 + 1, 304 * 32 + 1, 30001])
def test_ray_pe_edges(kind, n):
    """Encoding and its mlp2 term against 64 bits: an angle of up to 8 pi is
    off by 2^-24 of itself twice (FP32 pi, the product), 3e-6, and the term by
    that over its 27 inputs (3e-5 for weights of up to 0.3)."""
    from diver_gb300 import _native as N
    from diver_gb300.decoder import pack_plain, random_decoder

    dec = random_decoder(kind, 32, n)
    d = torch.randn(n, 3, generator=torch.Generator().manual_seed(n))
    d = d / d.norm(dim=-1, keepdim=True)
    dd, dp = d.cuda().contiguous(), pack_plain(dec).cuda()
    feat, out = torch.full((n + 1, 28), -7.0, device="cuda"), torch.full((n + 1, dec.width), -7.0, device="cuda")
    N.call("dv_ray_pe", int(kind[5:]), 32, N.ptr(dp), n, N.ptr(dd), N.ptr(feat), N.ptr(out), N.stream(dd.device))
    pe = torch_ref.pos_enc(d.double())
    w, b = dec.layers[dec.n_mlp1]
    ref = pe @ w.double()[:, dec.width:].t() + b.double()
    assert (feat[:n, :27].cpu().double() - pe).abs().max() <= 5e-6
    assert (out[:n].cpu().double() - ref).abs().max() <= 3e-5
    assert bool((feat[n:] == -7.0).all()) and bool((out[n:] == -7.0).all())
