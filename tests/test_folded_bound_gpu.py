"""GPU: the backwards that take mlp1's output layer WH and mlp2's first layer W2
as one matrix, where the hidden layer hid = WH^T A2 + bh is small against its
two parts.  With GF = A2^T delta,
    dL/dW2 = WH^T GF + bh (sum delta)^T,   dL/dWH = GF W2^T,
so rounding stands against the parts and not against hid.  Roundings of
different segments are independent and delta's signs are random, so sums over
segments and their errors grow by squares: with q = sqrt(sum over segments of
A2^2 delta^2),
    |error of dL/dW2| <= 2 eps Q2,  Q2 = |WH|^T q + |bh| sqrt(sum delta^2),
    |error of dL/dWH| <= 2 eps QH,  QH = q |W2|^T,
in Frobenius norms (2: the accumulators' partial sums in units of q).  eps, over
1000 segments:
  split  2^-16: an operand's two BF16 terms leave 2^-18 of it, a product 2^-17;
         64 MMAs (8 tiles of 8) add to the accumulator with 2^-23 each, 2^-17
  plain  2^-17: 32 segments and 32 atomic sums of 2^-24 each, 2^-18, and 32
         terms of the two layers' product, 2^-19
The decoder's ReLUs of mlp2 stay open (biases of 6), and mlp1's second hidden
layer is `base` and a little (biases of base), which bh takes away again: the
parts are about 26 base times hid."""
import pytest
import torch

from oracle import torch_ref
from tests.test_decode_plain_tiles_gpu import case
from tests.test_decode_tc_tiles_gpu import Lists

pytestmark = pytest.mark.gpu
N_SEG = 1000
EPS = {"split": 2.0 ** -16, "plain": 2.0 ** -17}


@pytest.mark.parametrize("form", ["split", "plain"])
@pytest.mark.parametrize("base", [0.0, 1.0, 8.0, 64.0])
@pytest.mark.parametrize("seed", [1, 2])
def test_error_of_the_folded_layers(form, base, seed):
    from diver_gb300 import _native as N
    from diver_gb300.decoder import pack_plain, unpack_plain_grad
    from diver_gb300.renderer import TcWeights

    vox, seg, ray, dirs, dec, d4 = case(N_SEG, 32, "diver32", seed)
    vox, L, W = vox / 6, dec.layers, 32
    L[1] = (L[1][0], torch.full((W,), base))
    b = L[2][1].clone()
    b[1:] = -(L[2][0][1:].double().sum(1) * base).float()
    L[2], L[3] = (L[2][0], b), (L[3][0], L[3][1] + 6.0)

    dv, ds, dr, dd, dp, dg = (x.cuda().contiguous() for x in (vox, seg, ray, dirs, pack_plain(dec), d4))
    st = N.stream(dv.device)
    pe = torch.empty(len(dd), 28, device="cuda"), torch.empty(len(dd), W, device="cuda")
    N.call("dv_ray_pe", 32, 32, N.ptr(dp), len(dd), N.ptr(dd), N.ptr(pe[0]), N.ptr(pe[1]), st)
    gv, gp = torch.zeros_like(dv), torch.zeros_like(dp)
    if form == "plain":
        N.call("dv_decode_bwd", 32, 32, N.ptr(dp), N.ptr(dv), 10, 8, 6, N.ptr(ds), N.ptr(dr), N_SEG, None, N.ptr(pe[0]),
               N.ptr(pe[1]), N.ptr(dg), N.ptr(gv), N.ptr(gp), st)
    else:
        tw, lists = TcWeights.from_decoder(dec, "cuda", mode="bf16s"), Lists(ds, dr)
        out4, save = torch.empty(N_SEG, 4, device="cuda"), tw.save_buffer(32, 32, N_SEG, "cuda")
        tw.decode(32, 32, dv, lists, pe[1], out4, st, None, save)
        assert tw.backward(32, dv, lists, *pe, dg, gv, gp, st, save, out4)
        assert int(tw.err.item()) == 0
    (gh, _), (g2, _) = unpack_plain_grad("diver32", 32, gp.cpu().double())[2:4]

    layers = [(w.double().requires_grad_(True), b.double().requires_grad_(True)) for w, b in L]
    feat = torch_ref.integrate(vox.double(), seg[:, :3].double(), seg[:, 3:].double(), per_axis=True)
    sigma, rgb = torch_ref.decode(layers, dec.n_mlp1, feat, dirs.double()[ray.long()])
    (torch.cat([sigma[:, None], rgb], 1) * d4.double()).sum().backward()
    with torch.no_grad():
        a2 = ((feat @ layers[0][0].t() + layers[0][1]).relu() @ layers[1][0].t() + layers[1][1]).relu()
        z = d4[:, 1:].double() * rgb * (1 - rgb)
        delta = z @ layers[4][0]  # mlp2's first activation is positive everywhere
        wh, w2, bh = layers[2][0][1:].abs(), layers[3][0][:, :W].abs(), layers[2][1][1:].abs()
        q = (a2.square().t() @ delta.square()).sqrt()  # [i][j]
        q2 = wh @ q + bh[:, None] * delta.square().sum(0).sqrt()  # [h][j]
        qh = q @ w2  # [i][h]
    assert float((g2[:, :W] - layers[3][0].grad[:, :W]).norm()) <= 2 * EPS[form] * float(q2.norm())
    assert float((gh[1:] - layers[2][0].grad[1:]).norm()) <= 2 * EPS[form] * float(qh.norm())
