"""Pin the CPU oracle against outputs of the reference's own Python (tests/golden)."""
import os

import pytest
import torch

from oracle import fakequant, kernel_path as kp

GOLD = torch.load(os.path.join(os.path.dirname(__file__), "golden", "reference_python.pt"), weights_only=False)


def test_pack_to_i4_matches_reference():
    g = GOLD["pack"]
    assert torch.equal(kp.pack_to_i4(g["vals"]), g["packed"])
    assert torch.equal(kp.two_compl(g["vals"], 4), g["two_compl"])
    assert torch.equal(kp.unpack_i4(g["packed"]), g["vals"])


@pytest.mark.parametrize("idx", range(len(GOLD["from_float"])))
def test_from_float_buffers_match_reference(idx):
    c = GOLD["from_float"][idx]
    buf = kp.from_float_buffers(c["weight"], c["scales"], c["fp_indices"], c["bits"], bias=c["bias"])
    ref = c["buffers"]
    for name in ("weights_scales", "int_weight", "reduced_w", "int_indices", "fp_indices"):
        assert torch.equal(buf[name], ref[name]), name
    if "fp_weight" in ref:
        assert torch.equal(buf["fp_weight"], ref["fp_weight"])
    assert (buf["bias"] is None) == c["bias_is_none"]
    if buf["bias"] is not None:
        assert torch.equal(buf["bias"], ref["bias"])


@pytest.mark.parametrize("idx", range(len(GOLD["fakequant"])))
def test_fakequant_port_matches_reference(idx):
    c = GOLD["fakequant"][idx]
    layer_probe = fakequant.FakeQuantLinear(torch.empty(0), c["act_scales"], c["nfp"], c["bits"])
    int_cols = layer_probe.q_idx
    scale = fakequant.weight_rtn_params(c["w"][:, int_cols], c["bits"], clip=True)
    assert torch.equal(scale, c["w_scale"])
    w_dq = c["w"].clone()
    w_dq[:, int_cols] = fakequant.weight_rtn_quantize(c["w"][:, int_cols], scale, c["bits"])
    assert torch.equal(w_dq, c["w_dq"])
    layer = fakequant.FakeQuantLinear(w_dq.half(), c["act_scales"], c["nfp"], c["bits"])
    with torch.no_grad():
        y = layer(c["x"])
    # The last step is torch's own fp16 linear on the host, whose order of summation depends on the CPU.  From the exact inputs of
    # that step (activations as quantized here, weights as above) the product is known in 64 bits, and any order of its K fp32
    # terms stays within K 2^-24 of the sum of their magnitudes before the one rounding to fp16 (2^-11 of the value, 2^-25 at
    # least).  The stored output has to lie there, too, which pins the activation path: a single activation one step of its grid
    # off moves some output by at least 13 bounds (4 bits) or 7 (8 bits without outliers; with outliers in the row, whose
    # products set the bound, by 2 and more for 91 % of the activations).
    xq, w = layer.linear_input(c["x"]).double(), layer.weight.double()
    exact = xq @ w.t()
    terms = xq.abs() @ w.abs().t()
    bound = 1.01 * xq.shape[-1] * 2.0 ** -24 * terms + exact.abs() * 2.0 ** -11 + 2.0 ** -25
    assert y.dtype == c["y"].dtype and y.shape == c["y"].shape
    assert bool(((y.double() - exact).abs() <= bound).all())
    assert bool(((c["y"].double() - exact).abs() <= bound).all())
