"""DualQuant's offline scale search (block coordinate descent) and final block quantisation,
batched over the column blocks of a weight (dualquant_b200/bcd.py), against vectors recorded from
the reference's wrap_dualquant_layer (layer_wrapper_dualquant.py:423-533, CPU, block after block).

Floating point: the batched form sums in another order than the reference's per-block loop, so the
bar is a tolerance - scales and stored weights within 2e-6 relative (measured 4e-7; the E8M0 and
column-only configurations come out bit-identical)."""
import os

import numpy as np
import pytest
import torch

from dualquant_b200 import bcd

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "reference_vectors.npz")
CFGS = {
    "iter15": dict(scale_option="row_column", row_init="max_abs", col_init="l1_norm", num_iter=15, scale_format="none"),
    "e4m3": dict(scale_option="row_column", row_init="max_abs", col_init="l2_norm", num_iter=5, scale_format="e4m3"),
    "e8m0": dict(scale_option="row_column", row_init="max_abs", col_init="l1_norm", num_iter=5, scale_format="e8m0"),
    "colonly": dict(scale_option="only_column", row_init="max_abs", col_init="l1_norm", num_iter=5, scale_format="none"),
}
RTOL = 2e-6


@pytest.fixture(scope="module")
def vec():
    return np.load(GOLDEN)


def _check(mat_q, cs, vec, tag):
    gm = torch.from_numpy(vec[f"bcd_{tag}_matq"])
    gc = torch.from_numpy(vec[f"bcd_{tag}_colscales"])
    assert mat_q.shape == gm.shape and cs.shape == gc.shape
    assert ((mat_q.cpu() - gm).abs().max() / gm.abs().max()).item() < RTOL
    assert ((cs.cpu() - gc).abs() / gc.abs()).max().item() < RTOL


@pytest.mark.parametrize("tag", sorted(CFGS))
def test_matches_reference_on_cpu(vec, tag):
    W = torch.from_numpy(vec["bcd_w"])
    mat_q, cs = bcd.dualquant_weight(W, block_size=128, **CFGS[tag])
    _check(mat_q, cs, vec, tag)
    if tag in ("e8m0", "colonly"):  # no unrounded row scale in the loop: bit-identical
        assert torch.equal(mat_q, torch.from_numpy(vec[f"bcd_{tag}_matq"]))


def test_wrap_dualquant_layer_is_a_drop_in(vec):
    W = torch.from_numpy(vec["bcd_w"])
    cfg = dict(num_splits=1, block_size=128, dualquant_to_element_tensor=True, **CFGS["e8m0"])
    lin = torch.nn.Linear(256, 96, bias=False)
    lin.weight.data.copy_(W)
    cs = bcd.wrap_dualquant_layer(lin, cfg, "rtn_int4", act_quant_flag=True)
    _check(lin.weight.data, cs, vec, "e8m0")
    # without activation quantisation the column scales are folded back into the stored weight
    lin2 = torch.nn.Linear(256, 96, bias=False)
    lin2.weight.data.copy_(W)
    assert bcd.wrap_dualquant_layer(lin2, cfg, "rtn_int4", act_quant_flag=False) is None
    assert torch.allclose(lin2.weight.data, lin.weight.data * cs.unsqueeze(0), rtol=1e-6, atol=0)


def test_search_lowers_the_reconstruction_error(vec):
    """What the search is for: W ~ mat_q * column_scales is closer to W than plain group-RTN."""
    W = torch.from_numpy(vec["bcd_w"])
    W3 = W.reshape(96, 2, 128)
    s = W3.abs().amax(dim=-1, keepdim=True) / 7.0
    rtn = ((W3 / s).round().clamp(-8, 7) * s).reshape(96, 256)
    mat_q, cs = bcd.dualquant_weight(W, block_size=128, **CFGS["iter15"])
    assert ((mat_q * cs - W) ** 2).mean() < 0.9 * ((rtn - W) ** 2).mean()


def test_unsupported_options_say_so():
    W = torch.randn(8, 128)
    with pytest.raises(NotImplementedError):
        bcd.dualquant_weight(W, quant_method="nvfp4")
    with pytest.raises(NotImplementedError):
        bcd.dualquant_weight(W, scale_format="e5m3")
    with pytest.raises(ValueError):
        bcd.dualquant_weight(W, block_size=96)
    with pytest.raises(ValueError):
        bcd.dualquant_weight(W, scale_option="both")


@pytest.mark.gpu
@pytest.mark.parametrize("tag", sorted(CFGS))
def test_matches_reference_on_the_gpu_and_packs(vec, tag):
    """The same search on the device, then DualQuant's outputs -> packed int4 artefact -> W4A4 linear:
    the stored weight lies on the int4 group grid, so packing it loses nothing."""
    from dualquant_b200 import _lib, ops, wrap
    from oracle import dq_oracle as O

    dev = "cuda:0"
    W = torch.from_numpy(vec["bcd_w"])
    mat_q, cs = bcd.dualquant_weight(W.to(dev), block_size=128, **CFGS[tag])
    _check(mat_q, cs, vec, tag)
    pw, a = wrap.pack_from_dualquant(mat_q, cs)
    x = torch.randn(24, 256, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16)
    y = ops.linear_w4a4_int4(x.to(dev), a, None, pw, None, scale_fp16=False)
    _lib.device_status(0)
    qx, sx, _ = O.quant_act_int4(x, cs.cpu(), None, False)
    qw, sw = O.quant_w_int4(mat_q.cpu().to(torch.bfloat16))
    ref = O.dequant_matmul(qx, sx, qw, sw, None)
    assert ((y.cpu().double() - ref).abs().max() / ref.abs().max()).item() < 1e-5
    # the artefact's codes x fp16 group scales reproduce the stored weight to its bf16 storage
    # rounding (2^-8 relative; the reference keeps mat_q in the layer's bf16 weight as well)
    back = O.dequant_w(qw, sw)
    assert ((back - mat_q.cpu()).abs().max() / mat_q.abs().max().cpu()).item() < 6e-3


@pytest.mark.gpu
def test_full_size_layer_on_the_gpu():
    """A 4096 x 4096 weight (32 column blocks searched at once): finite scales, lower error than
    group-RTN, and every block equal to the same block searched on its own."""
    dev = "cuda:0"
    g = torch.Generator(device=dev).manual_seed(5)
    W = torch.randn(4096, 4096, generator=g, device=dev) * 0.02
    W[:, torch.randperm(4096, generator=g, device=dev)[:40]] *= 10
    cfg = CFGS["e8m0"]
    mat_q, cs = bcd.dualquant_weight(W, block_size=128, **cfg)
    assert torch.isfinite(mat_q).all() and torch.isfinite(cs).all()
    W3 = W.reshape(4096, 32, 128)
    s = W3.abs().amax(dim=-1, keepdim=True) / 7.0
    rtn = ((W3 / s).round().clamp(-8, 7) * s).reshape(4096, 4096)
    assert ((mat_q * cs - W) ** 2).mean() < ((rtn - W) ** 2).mean()
    for b in (0, 17, 31):
        mq_b, cs_b = bcd.dualquant_weight(W[:, b * 128:(b + 1) * 128].contiguous(), block_size=128, **cfg)
        assert torch.allclose(mq_b, mat_q[:, b * 128:(b + 1) * 128], rtol=1e-5, atol=1e-9)
        assert torch.allclose(cs_b, cs[b * 128:(b + 1) * 128], rtol=1e-5, atol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols,bs", [(1, 128, 128), (7, 256, 32), (33, 192, 64), (130, 512, 256), (1025, 384, 128)])
@pytest.mark.parametrize("option", ["row_column", "only_column", "only_row"])
@pytest.mark.parametrize("fmt", ["none", "e8m0", "e4m3"])
def test_search_kernels_against_the_tensor_form(rows, cols, bs, option, fmt):
    """Ragged row counts (chunk and warp remainders) and every block size: one iteration agrees with the tensor
    expressions on the CPU to the order of fp32 sums (more iterations would compare a scale or code that stepped at
    a rounding boundary); the fused quantise-and-pack gives the bytes of the two separate steps."""
    from dualquant_b200 import ops, wrap

    g = torch.Generator().manual_seed(rows + cols)
    W = torch.randn(rows, cols, generator=g) * 0.02
    for col_init, row_init in (("l1_norm", "max_abs"), ("l2_norm", "max_abs"), ("max_abs", "all_one"), ("all_one", "max_abs")):
        cfg = dict(block_size=bs, num_iter=1, scale_option=option, row_init=row_init, col_init=col_init, scale_format=fmt)
        ref_q, ref_c = bcd.dualquant_weight(W, **cfg)
        ref_a, ref_b = bcd.dualquant_scales(W, **cfg)
        mat_q, cs = bcd.dualquant_weight(W.cuda(), **cfg)
        alpha, beta = bcd.dualquant_scales(W.cuda(), **cfg)
        for got, ref in ((alpha, ref_a), (beta, ref_b), (cs, ref_c)):
            assert got.shape == ref.shape
            off = (got.cpu() - ref).abs() > 1e-5 * ref.abs()
            assert torch.equal(torch.isfinite(got.cpu()), torch.isfinite(ref))
            assert (off & torch.isfinite(ref)).float().mean() <= (0.02 if rows > 1 else 0.1)
        same = torch.isfinite(ref_q)
        assert torch.equal(torch.isfinite(mat_q.cpu()), same)  # a column whose codes are all zero has no scale
        bad = (mat_q.cpu() - ref_q).abs()[same] > 1e-4 * ref_q.abs().nan_to_num(0.0, 0.0, 0.0).max()
        assert bad.numel() == 0 or bad.float().mean() < 0.02
    if cols % 128 == 0:
        mat_q = W.cuda()
        for w in (mat_q, mat_q.to(torch.bfloat16)):
            a, b = ops.quant_pack_w_int4(w), ops.pack_w_int4(*ops.quant_w_int4(w))
            assert torch.equal(a.w_packed, b.w_packed) and torch.equal(a.sw_t.view(torch.int16), b.sw_t.view(torch.int16))
        assert torch.equal(wrap.pack_from_dualquant(mat_q)[0].w_packed, a.w_packed)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(1000, 1024), (4096, 1024), (8192, 256)])
def test_column_sums_are_as_close_to_64_bits_as_a_tensor_reduction(rows, cols):
    """One iteration against the same steps in 64 bits.  A column scale is a quotient of two sums over all rows, each
    rounded at the last addition (2^-25 of it on average) after chains of some ten roundings: half the columns stay
    within 2^-24.  Adding the 32 partial sums in order took the median to 1.5 x 2^-24."""
    bs = 128
    W = torch.randn(rows, cols, generator=torch.Generator().manual_seed(rows)).cuda() * 0.02
    alpha, beta = bcd.dualquant_scales(W, block_size=bs, num_iter=1)
    W3 = W.double().view(rows, cols // bs, bs)
    b = 1.0 / W3.abs().sum(0)
    a = 7.0 / (W3 * b).abs().amax(-1)
    m = (a.unsqueeze(-1) * W3 * b).round().clamp(-8, 7) / b
    a_inv = (W3 * m).sum(-1) / (m ** 2).sum(-1)
    m = (W3 * b / a_inv.unsqueeze(-1)).round().clamp(-8, 7) * a_inv.unsqueeze(-1)
    b = (m ** 2).sum(0) / (W3 * m).sum(0)
    assert ((alpha.double() * a_inv) - 1).abs().median().item() < 2.0 ** -24
    assert ((beta.double() / b) - 1).abs().median().item() < 2.0 ** -24
