"""Products right behind an upload that nothing waits for (slai_qmatrix_create_from_device): they may start while the kernel in front of
them still runs and read their weights before they wait for it, so that kernel must not be the one that writes the weights."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from slai_b200 import synth
from slai_b200._lib import SlaiError
from slai_b200.ops import GpuQuantMatrix
from helpers import rel_l2

pytestmark = pytest.mark.gpu
RELAXED, PROGRAMMATIC, KERNEL_NODE = 2, 1, 0


class EdgeData(C.Structure):
    _fields_ = [("from_port", C.c_ubyte), ("to_port", C.c_ubyte), ("type", C.c_ubyte), ("reserved", C.c_ubyte * 5)]


class KernelParams(C.Structure):
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("shared", C.c_uint), ("args", C.c_void_p), ("extra", C.c_void_p),
                ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def captured_edges(backend, calls):
    """What `calls` puts into the context's stream, as (kernel in front, kernel behind, programmatic) per edge; nothing runs."""
    cu = C.CDLL("libcuda.so.1")

    def ok(rc):
        assert rc == 0, rc

    def name(node):
        kind = C.c_int()
        ok(cu.cuGraphNodeGetType(node, C.byref(kind)))
        if kind.value != KERNEL_NODE:
            return "copy or fill"
        p, s = KernelParams(), C.c_char_p()
        ok(cu.cuGraphKernelNodeGetParams_v2(node, C.byref(p)))
        ok(cu.cuFuncGetName(C.byref(s), C.c_void_p(p.func)) if p.func else cu.cuKernelGetName(C.byref(s), C.c_void_p(p.kern)))
        return s.value.decode()

    stream, graph = C.c_void_p(backend.lib.slai_ctx_stream(backend.h)), C.c_void_p()
    backend.synchronize()
    ok(cu.cuStreamBeginCapture_v2(stream, RELAXED))
    try:
        calls()
    finally:
        ok(cu.cuStreamEndCapture(stream, C.byref(graph)))
    n = C.c_size_t(0)
    ok(cu.cuGraphGetEdges_v2(graph, None, None, None, C.byref(n)))
    src, dst, data = (C.c_void_p * n.value)(), (C.c_void_p * n.value)(), (EdgeData * n.value)()
    ok(cu.cuGraphGetEdges_v2(graph, src, dst, data, C.byref(n)))
    edges = [(name(C.c_void_p(src[i])), name(C.c_void_p(dst[i])), data[i].type == PROGRAMMATIC) for i in range(n.value)]
    ok(cu.cuGraphDestroy(graph))
    return edges


@pytest.mark.parametrize("n_batch", [1, 3])
@pytest.mark.parametrize("fmt", [synth.FMT_F32, synth.FMT_Q4_1, synth.FMT_Q8_0, synth.FMT_Q4_K])
def test_no_early_start_behind_the_kernel_that_writes_the_weights(backend, ctx, fmt, n_batch):
    M, K = 64, 512
    rng = np.random.default_rng(fmt)
    raw = synth.quantize(fmt, synth.normal_matrix(fmt, M, K)) if fmt != synth.FMT_F32 else synth.normal_matrix(fmt, M, K)
    blocks = backend.vector(np.ascontiguousarray(raw).view(np.uint8).reshape(-1), np.uint8)
    vs, outs = backend.vector(rng.standard_normal(8 * K + 8).astype(np.float32)), backend.zeros(8 * M)
    v, out = vs.view(0, n_batch * K), outs.view(0, n_batch * M)
    warm = GpuQuantMatrix(backend, fmt, M, K, device_blocks=blocks.ptr, nbytes=blocks.nbytes)
    ctx.matmul_quant_assign(out, warm, v, n_batch=n_batch)  # scratch and kernel attributes are there before the recording
    made = []

    def calls():
        m = GpuQuantMatrix(backend, fmt, M, K, device_blocks=blocks.ptr, nbytes=blocks.nbytes)
        made.append(m)
        if fmt in (synth.FMT_Q8_0, synth.FMT_Q4_K):
            with pytest.raises(SlaiError):  # refused: it takes nothing away from the next one's order
                ctx.matmul_quant_assign(outs.view(0, 2 * M), m, vs.view(1, 2 * K), n_batch=2)
        ctx.matmul_quant_assign(out, m, v, n_batch=n_batch)

    edges = captured_edges(backend, calls)
    programmatic = [(a, b) for a, b, p in edges if p]
    assert programmatic or not any("gemv" in b for _, b, _ in edges), edges  # the overlap itself is there
    for a, _ in programmatic:
        assert "copy or fill" not in a and "place" not in a and "legacy" not in a, edges


@pytest.mark.parametrize("fmt", [synth.FMT_Q8_0, synth.FMT_Q4_K])
def test_products_right_behind_an_upload(backend, ctx, fmt):
    """Values, with everything in flight: upload, a product recorded for later, products at once."""
    M, K = 4096, 2048  # the upload takes several times a launch
    rng = np.random.default_rng(fmt)
    raw = synth.quantize(fmt, synth.normal_matrix(fmt, M, K))
    W = O.dequantize(fmt, raw).reshape(M, K).astype(np.float64)
    blocks = backend.vector(np.ascontiguousarray(raw).view(np.uint8).reshape(-1), np.uint8)
    x = rng.standard_normal((3, K)).astype(np.float32)
    v, one, three = backend.vector(x.ravel()), backend.zeros(M), backend.zeros(3 * M)
    warm = GpuQuantMatrix(backend, fmt, M, K, raw)
    ctx.matmul_quant_assign(one, warm, v.view(0, K))  # scratch and kernel attributes are there before the recording
    ctx.matmul_quant_assign(three, warm, v, n_batch=3)
    for first in (1, 3):
        m = GpuQuantMatrix(backend, fmt, M, K, device_blocks=blocks.ptr, nbytes=blocks.nbytes)
        with backend.record() as rec:
            ctx.matmul_quant_assign(one, m, v.view(0, K))
        for n_batch, out in ((1, one), (3, three)) if first == 1 else ((3, three), (1, one)):
            ctx.matmul_quant_assign(out, m, v.view(0, n_batch * K), n_batch=n_batch)
        # exact integers but for the vectors' 27 bits and one f32 sum of 8 or 16 terms: far below 2e-6
        assert rel_l2(one.to_numpy(), W @ x[0]) < 2e-6
        for b in range(3):
            assert rel_l2(three.to_numpy().reshape(3, M)[b], W @ x[b]) < 2e-6
        rec.launch()
        assert rel_l2(one.to_numpy(), W @ x[0]) < 2e-6
        rec.close()
