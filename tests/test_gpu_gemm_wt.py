"""GPU parity of the products with the weight rows on the M side of the MMA (csrc/tlc_gemm_wt.cu), at the edges of
their tiles: rows and columns around 16, 64, 128 and 256, K of one block, one step and more, every form."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TIGHT = 1e-3


@pytest.fixture(params=[0, 1, 3, 8, 9], ids=["auto", "ks1", "ks3", "ks8", "stream"])
def form(request, dev):
    """CTAs per tile of the cluster form, or 9: the stream form.  (Small products of 17 to 48 rows are the GEMV's by
    default.)"""
    dev.set_option("gemm_wt_ks", request.param)
    dev.set_option("gemm_min_m", 1)
    yield request.param
    dev.set_option("gemm_wt_ks", 0)
    dev.set_option("gemm_min_m", 0)


@pytest.mark.parametrize("qtype,n,k,m", [(2, 1, 64, 17), (2, 129, 96, 33), (8, 300, 2080, 130), (8, 127, 160, 257),
                                         (2, 400, 1376, 18), (1, 17, 72, 2), (1, 130, 200, 129), (1, 257, 77, 5)])
def test_linear_edges(dev, ref, form, qtype, n, k, m):
    from tensorlogic_b200 import synth
    from tensorlogic_b200.api import QTensor, linear
    x = synth.activations(3, f"wtx{m}x{k}", (m, k))
    bias = synth.activations(3, f"wtb{n}", (n,))
    if qtype == 1:
        w = (synth.normal(3, synth.tensor_id(f"wtw{n}x{k}"), (n, k)) * 0.05).astype(np.float16)
        want = ref.linear_f32acc(x, w)
    else:
        w = synth.blocks(qtype, 3, synth.tensor_id(f"wtw{n}x{k}"), n, k)
        want = ref.linear_q(qtype, w, n, k, x)
    got = linear(dev.tensor(x), QTensor.from_blocks(dev, qtype, n, k, w), dev.tensor(bias)).numpy()
    want = (want.astype(np.float16) + bias).astype(np.float16)
    assert got.shape == (m, n) and rel_l2(got, want) < TIGHT


@pytest.mark.parametrize("m,k,n", [(1, 8, 1), (17, 129, 65), (128, 64, 128), (129, 520, 136), (257, 72, 31)])
def test_matmul_edges(dev, ref, form, m, k, n):
    from tensorlogic_b200 import synth
    from tensorlogic_b200.api import matmul
    a, b = synth.activations(4, f"ma{m}x{k}", (m, k)), synth.activations(4, f"mb{k}x{n}", (k, n))
    got = matmul(dev.tensor(a), dev.tensor(b)).numpy()
    assert rel_l2(got, ref.linear_f32acc(a, np.ascontiguousarray(b.T))) < TIGHT


@pytest.mark.parametrize("qtype", [2, 8])
@pytest.mark.parametrize("m", [17, 150])
def test_fused_entry_points(dev, form, qtype, m):
    """Norm + three projections with RoPE, the SiLU.mul pair (ragged N) and the residual against the same
    operations one by one."""
    from tensorlogic_b200 import synth
    from tensorlogic_b200.api import QTensor, add, linear, linear_residual, norm_linear_multi, rms_norm, rope, swiglu, swiglu_gate_up
    k = 320
    def q(name, rows):
        return QTensor.synthetic(dev, qtype, rows, k, 5, synth.tensor_id(name), scale_log2=0 if qtype == 2 else -4)
    x, nw = dev.tensor(synth.activations(5, "fx", (m, k))), dev.tensor(synth.norm_weight(5, "fn", k))
    h = rms_norm(x, nw, 1e-5)
    ws = [q("fq", 256), q("fk", 128), q("fv", 128)]
    outs = norm_linear_multi(x, ws, nw, 1e-5, rope_heads=[4, 2, 0], position_offset=7)
    for y, w, heads in zip(outs, ws, (4, 2, 0)):
        want = linear(h, w)
        if heads:
            want = rope(want.reshape((m, heads, w.shape[0] // heads)), 7)
        assert rel_l2(y.numpy().ravel(), want.numpy().ravel()) < TIGHT
    g, u = q("fg", 200), q("fu", 200)
    assert rel_l2(swiglu_gate_up(x, g, u, nw, 1e-5).numpy(), swiglu(linear(h, g), linear(h, u)).numpy()) < 2e-3
    o = q("fo", 136)
    r = dev.tensor(synth.activations(5, "fr", (m, 136)))
    assert rel_l2(linear_residual(h, o, r).numpy(), add(linear(h, o), r).numpy()) < TIGHT
