"""GPU parity of the fused GEMV for 2 to 16 activation rows (csrc/tlc_gemv_kernel.cuh) where its split of K changes:
eight and sixteen warps, one to three windows a warp, clusters, and rows and columns that fill nothing."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TIGHT = 1e-3


@pytest.mark.parametrize("qtype", [2, 8])
@pytest.mark.parametrize("n,k", [(16, 32), (17, 1056), (40, 3072), (33, 3104), (50, 4128), (48, 6176), (100, 12320)])
@pytest.mark.parametrize("m", [2, 8, 9, 16])
def test_rows_and_windows(dev, ref, qtype, n, k, m):
    from tensorlogic_b200 import synth
    from tensorlogic_b200.api import QTensor, linear
    raw = synth.blocks(qtype, 6, synth.tensor_id(f"gr{n}x{k}"), n, k)
    x = synth.activations(6, f"gx{m}x{k}", (m, k))
    got = linear(dev.tensor(x), QTensor.from_blocks(dev, qtype, n, k, raw)).numpy()
    assert rel_l2(got, ref.linear_q(qtype, raw, n, k, x)) < TIGHT


@pytest.mark.parametrize("qtype", [2, 8])
@pytest.mark.parametrize("k", [2048, 8256])
@pytest.mark.parametrize("m", [3, 16])
def test_fused_epilogues(dev, qtype, k, m):
    """Norm + projections with RoPE, the SiLU.mul pair over more slabs than one round, the residual, against the
    operations one by one."""
    from tensorlogic_b200 import synth
    from tensorlogic_b200.api import (QTensor, add, linear, linear_residual, norm_linear_multi, rms_norm, rope, swiglu,
                                      swiglu_gate_up)
    def q(name, rows):
        return QTensor.synthetic(dev, qtype, rows, k, 8, synth.tensor_id(name), scale_log2=-1 if qtype == 2 else -5)
    x, nw = dev.tensor(synth.activations(8, f"ex{k}", (m, k))), dev.tensor(synth.norm_weight(8, f"en{k}", k))
    h = rms_norm(x, nw, 1e-5)
    ws = [q("eq", 192), q("ek", 64), q("ev", 64)]
    outs = norm_linear_multi(x, ws, nw, 1e-5, rope_heads=[3, 1, 0], position_offset=11)
    for y, w, heads in zip(outs, ws, (3, 1, 0)):
        want = linear(h, w)
        if heads:
            want = rope(want.reshape((m, heads, 64)), 11)
        assert rel_l2(y.numpy().ravel(), want.numpy().ravel()) < TIGHT
    g, u = q("eg", 1000), q("eu", 1000)
    assert rel_l2(swiglu_gate_up(x, g, u, nw, 1e-5).numpy(), swiglu(linear(h, g), linear(h, u)).numpy()) < 2e-3
    r = dev.tensor(synth.activations(8, "er", (m, 1000)))
    assert rel_l2(linear_residual(h, g, r).numpy(), add(linear(h, g), r).numpy()) < TIGHT


@pytest.mark.parametrize("n,k,m", [(16, 256, 1), (15, 2304, 8), (33, 4096, 9), (40, 4352, 16), (17, 8448, 2), (50, 2048, 40)])
def test_q6_k_windows(dev, ref, n, k, m):
    """Q6_K on the same kernel: one super-block a warp, eight and sixteen warps, clusters, further passes."""
    from tensorlogic_b200 import synth
    from tensorlogic_b200.api import QTensor, linear
    rng = np.random.default_rng(n * k + m)
    raw = rng.integers(0, 256, (n * k // 256, 210), dtype=np.uint8)
    raw[:, 208:210] = rng.uniform(-2e-5, 2e-5, (raw.shape[0], 1)).astype(np.float16).view(np.uint8)
    x = synth.activations(9, f"q6x{m}x{k}", (m, k))
    got = linear(dev.tensor(x), QTensor.from_blocks(dev, 14, n, k, raw)).numpy()
    assert rel_l2(got, ref.linear_q(14, raw.reshape(-1), n, k, x)) < TIGHT


def _exact_product(qtype, raw, x):
    """x . W^T in 64 bits with the weights d * (q - 8) as the blocks define them, rounded once to f16."""
    d = raw[..., :2].copy().view(np.float16).astype(np.float64)
    if qtype == 2:
        q = np.concatenate([(raw[..., 2:] & 15).astype(np.float64), (raw[..., 2:] >> 4).astype(np.float64)], -1) - 8
    else:
        q = raw[..., 2:].view(np.int8).astype(np.float64)
    return (x.astype(np.float64) @ (q * d).reshape(raw.shape[0], -1).T).astype(np.float16)


@pytest.mark.parametrize("qtype", [2, 8])
@pytest.mark.parametrize("m,n,k", [(2, 200, 2048), (9, 200, 11008), (16, 200, 8192), (12, 100, 28672), (17, 300, 64),
                                   (33, 4100, 1216), (48, 9344, 1504)])
def test_weights_are_not_rounded(dev, qtype, m, n, k):
    """Up to sixteen rows, and up to 48 of a short K, d * (q - 8) is multiplied as it is.  The f32 sum of K terms is then off by about 1e-6 of the
    output, which moves about one in a hundred of the roundings to f16 (steps of 5e-4 to 1e-3); weights rounded to
    f16 first, each by up to 2^-11, would move about four in ten."""
    from tensorlogic_b200 import synth
    from tensorlogic_b200.api import QTensor, linear
    raw = synth.blocks(qtype, 7, synth.tensor_id(f"nr{n}x{k}"), n, k, scale_log2=-3 if qtype == 2 else -7)
    x = synth.activations(7, f"nx{m}x{k}", (m, k))
    got = linear(dev.tensor(x), QTensor.from_blocks(dev, qtype, n, k, raw)).numpy()
    assert np.mean(got == _exact_product(qtype, raw, x)) > 0.95


@pytest.mark.parametrize("qtype", [2, 8])
@pytest.mark.parametrize("m,k", [(9, 65536), (16, 65664), (8, 98304), (9, 98304), (9, 98432), (16, 98432)])
def test_longest_rows(dev, ref, qtype, m, k):
    """K where sixteen rows no longer fit one launch, where eight do not, and beyond."""
    from tensorlogic_b200 import synth
    from tensorlogic_b200.api import QTensor, linear
    n = 20
    raw = synth.blocks(qtype, 6, synth.tensor_id(f"lr{k}"), n, k, scale_log2=-3 if qtype == 2 else -7)
    x = synth.activations(6, f"lx{m}x{k}", (m, k))
    got = linear(dev.tensor(x), QTensor.from_blocks(dev, qtype, n, k, raw)).numpy()
    assert rel_l2(got, ref.linear_q(qtype, raw, n, k, x)) < TIGHT
