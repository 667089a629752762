"""The builtins are launched dependent: a kernel may be resident, and past everything it does before its dependency
wait, while the one in front of it still stores.  What a program has just computed must not be read that early.  Each
program below is queued behind work that keeps the GPU busy, with all operands on the device (an upload in between
would order the kernels by itself), and gives the bits that it gives with dependent launch off."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _both(dev, program):
    """The program's results with dependent launch on and off: lists of arrays."""
    got = []
    for pdl in (1, 0):
        dev.set_option("pdl", pdl)
        try:
            got.append([t.numpy() for t in program()])
        finally:
            dev.set_option("pdl", 1)
    return got


def _busy(dev):
    """A few products of some ten microseconds: the host runs ahead of the GPU from here on."""
    from tensorlogic_b200.api import matmul
    a = dev.tensor(np.ones((2048, 2048), np.float16))

    def queue():
        for _ in range(8):
            matmul(a, a)
    return queue


@pytest.mark.parametrize("H,Hkv,D", [(32, 4, 64), (8, 1, 128), (8, 8, 64)])
@pytest.mark.parametrize("rows", [100, 640, 2000])
def test_attention_right_after_append(dev, H, Hkv, D, rows):
    """One query at the last of the rows that the append in front of it stores: none of them is there before."""
    from tensorlogic_b200.api import KVCache
    rng = np.random.default_rng(rows + D)
    normal = lambda *shape: dev.tensor(rng.standard_normal(shape).astype(np.float16))
    sets = [(normal(rows, Hkv, D), normal(rows, Hkv, D)) for _ in range(3)]
    q, cache, queue = normal(1, H, D), KVCache(dev, 1, Hkv, D, max_seq=2048), _busy(dev)

    def program():
        out = []
        for k, v in sets * 4:
            queue()
            cache.lengths[0] = 0
            cache.append(0, k, v)
            out.append(cache.attention(0, q, H, q_pos0=rows - 1))
        return out

    on, off = _both(dev, program)
    for i, (a, b) in enumerate(zip(on, off)):
        assert np.array_equal(a.view(np.uint16), b.view(np.uint16)), i


@pytest.mark.parametrize("m", [1, 5, 16, 40])
@pytest.mark.parametrize("qtype", [1, 2, 8, 14])
def test_norm_weights_computed_right_before(dev, qtype, m):
    """mul -> norm_linear_multi and mul -> swiglu_gate_up: the norm weights are the product, in every form that norms
    (one row, two to sixteen, the GEMM, dense and Q6_K weights)."""
    from tensorlogic_b200 import synth
    from tensorlogic_b200.api import QTensor, mul, norm_linear_multi, swiglu_gate_up
    k, n = 8192, 96
    rng = np.random.default_rng(qtype + m)
    if qtype == 14:
        raw = rng.integers(0, 256, (n * k // 256, 210), dtype=np.uint8)
        raw[:, 208:210] = rng.uniform(1e-5, 2e-5, (raw.shape[0], 1)).astype(np.float16).view(np.uint8)
        w = QTensor.from_blocks(dev, 14, n, k, raw)
    elif qtype == 1:
        w = QTensor.normal_f16(dev, n, k, 3, synth.tensor_id("dw"), 0.0, 0.02)
    else:
        w = QTensor.synthetic(dev, qtype, n, k, 3, synth.tensor_id("dw"), scale_log2=-3 if qtype == 2 else -7)
    normal = lambda *shape: dev.tensor(rng.standard_normal(shape).astype(np.float16))
    x, norms, scale, queue = normal(m, k), [normal(k) for _ in range(3)], normal(k), _busy(dev)

    def program():
        out = []
        for nw in norms * 4:
            queue()
            out += norm_linear_multi(x, [w], mul(nw, scale), 1e-5)
            if qtype in (2, 8):
                queue()
                out.append(swiglu_gate_up(x, w, w, mul(nw, scale), 1e-5))
        return out

    on, off = _both(dev, program)
    for i, (a, b) in enumerate(zip(on, off)):
        assert np.array_equal(a.view(np.uint16), b.view(np.uint16)), i


def test_generated_weights_are_there_when_their_handle_is(dev):
    """Kernels fetch weights and a model's norm weights in front of their dependency wait: nothing that writes them
    may be in flight once the call that creates them has returned."""
    import torch
    from tensorlogic_b200 import synth
    from tensorlogic_b200.api import QTensor
    stream = torch.cuda.ExternalStream(dev.stream)
    queue = _busy(dev)
    for make in (lambda: QTensor.synthetic(dev, 2, 8192, 28672, 1, synth.tensor_id("g4")),
                 lambda: QTensor.synthetic(dev, 8, 8192, 28672, 1, synth.tensor_id("g8")),
                 lambda: QTensor.normal_f16(dev, 8192, 8192, 1, synth.tensor_id("gf"), 1.0, 0.02)):
        queue()
        w = make()
        assert stream.query()
        del w
