"""The quantizer's assignment step on the device (hlq_quantize_with_scales_device) against the
reference's own outputs (golden fixtures made with GPTQ/quant.py) and the oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from conftest import golden_cases, load_golden  # noqa: E402
from elutq_b200 import _lib, format as F  # noqa: E402
from oracle import hlq_oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", golden_cases())
def test_device_quantizer_matches_the_reference_fixture(name):
    d = load_golden(name)
    n, k, g, q = d["n"], d["k"], d["g"], d["q"]
    s16 = d["w_scale_f32"].astype(np.float16).astype(np.float32).reshape(n * (k // g), q)
    z16 = d["w_zero_f32"].astype(np.float16).astype(np.float32).reshape(n * (k // g))
    got = F.quantize_with_scales_device(torch.from_numpy(d["requant_in"]).cuda(), torch.from_numpy(s16).cuda(),
                                        torch.from_numpy(z16).cuda()).cpu().numpy()
    # the restatement: same fp32 arithmetic up to the order in which a combination's scales are
    # added, so the same choice everywhere but at exact near-ties
    assert (got == O.quantize_with_scales(d["requant_in"], s16, z16, q)).all(axis=2).mean() > 0.9999
    # the reference itself (torch.matmul may sum the scales in another order: ties can differ)
    same = (got == d["requant_out"]).all(axis=2)
    assert same.mean() > 0.999
    np.testing.assert_allclose(O.dequantize_with_scales(got, s16, z16),
                               O.dequantize_with_scales(d["requant_out"], s16, z16), atol=1e-6)


@pytest.mark.parametrize("q,g,blocks", [(1, 128, 7), (2, 64, 1000), (3, 128, 333), (4, 32, 4096)])
def test_device_quantizer_equals_oracle_and_feeds_the_export(q, g, blocks):
    rng = np.random.default_rng(q * 100 + g)
    w = (0.03 * rng.standard_normal((blocks, g))).astype(np.float32)
    s = (0.02 * rng.standard_normal((blocks, q))).astype(np.float32)        # alternating mode: signs are free
    z = (0.01 * rng.standard_normal(blocks)).astype(np.float32)
    got = F.quantize_with_scales_device(torch.from_numpy(w).cuda(), torch.from_numpy(s).cuda(),
                                        torch.from_numpy(z).cuda())
    ref = O.quantize_with_scales(w, s, z, q)
    got = got.cpu().numpy()
    assert (got == ref).all(axis=2).mean() > 0.9999
    # nearest: no other combination is closer than the chosen one
    back = O.dequantize_with_scales(got, s, z)
    combos = O.bit_combinations(q)
    allv = (s @ combos.T)[:, None, :] + z[:, None, None]
    assert (np.abs(back - w)[..., None] <= np.abs(allv - w[..., None]) + 1e-6).all()


def test_device_quantizer_argument_errors():
    w = torch.zeros((2, 8), device="cuda")
    with pytest.raises(ValueError):
        F.quantize_with_scales_device(w, torch.zeros((3, 2), device="cuda"), torch.zeros(2, device="cuda"))
    with pytest.raises(_lib.HlqError):
        F.quantize_with_scales_device(w, torch.zeros((2, 5), device="cuda"), torch.zeros(2, device="cuda"))
    with pytest.raises(RuntimeError):
        F.quantize_with_scales_device(torch.zeros((2, 8)), torch.zeros((2, 2)), torch.zeros(2))


# group sizes of the register kernel (few blocks: eight lanes a group; many: four) and one of the general kernel
@pytest.mark.parametrize("q", [1, 2, 3, 4])
@pytest.mark.parametrize("g,blocks", [(32, 1), (32, 1003), (32, 76001), (64, 77), (64, 76001), (128, 5), (128, 76001), (48, 65)])
def test_one_pass_quantizer_is_fit_plus_assignment(q, g, blocks):
    rng = np.random.default_rng(q * 1000 + g + blocks)
    w = (0.02 * rng.standard_normal((blocks, g))).astype(np.float32)
    w[0] = 0.25                                             # a constant block: singular system, exact result
    if blocks > 3:
        w[2] = np.where(rng.random(g) < 0.5, -0.5, 0.5)     # two values only: planes without weights
    wd = torch.from_numpy(w).cuda()
    rec, quant, s, z = F.pseudo_quantize_device(wd.reshape(blocks, g), q, g)
    s, z = s.reshape(blocks, q), z.reshape(blocks)
    # assignment and reconstruction are exactly those of the returned scales
    again = F.quantize_with_scales_device(wd, s, z)
    assert torch.equal(quant.reshape(blocks, g, q), again)
    want = torch.zeros((blocks, g), device="cuda")
    for j in range(q):
        want = want + again[..., j].float() * s[:, j:j + 1]
    assert torch.equal(rec, want + z[:, None])
    s2, z2 = F.fit_alternating_device(wd, q)
    assert torch.equal(s, s2) and torch.equal(z, z2)
    assert float((rec[0] - 0.25).abs().max()) <= 1e-6
    # the fit against the oracle on the first and last blocks: the same where every assignment agrees; a
    # parted weight (equally far from two values) costs the same either way, so the errors agree everywhere
    pick = np.unique(np.r_[0:min(blocks, 40), max(0, blocks - 40):blocks])
    so, zo = O.fit_alternating(w[pick], q)
    bo = O.quantize_with_scales(w[pick], so, zo, q)
    err_o = ((w[pick] - O.dequantize_with_scales(bo, so, zo)) ** 2).mean()
    err = ((w[pick] - rec.cpu().numpy()[pick]) ** 2).mean()
    assert abs(err - err_o) <= 1e-5 * err_o + 1e-14
    same = (again.cpu().numpy()[pick] == bo).all(axis=(1, 2))
    same[0] = False                                         # the constant block's planes are arbitrary
    assert same.sum() >= 0.9 * (len(pick) - 2)
    np.testing.assert_allclose(s.cpu().numpy()[pick][same], so[same], rtol=2e-4, atol=1e-7)
