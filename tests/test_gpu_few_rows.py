"""Inference on few rows per expert: when its GEMMs may begin early, which calls take them, and their edges."""
import ctypes

import pytest
import torch

from oracle import quant as Q

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from sonicmoe import ops as _ops
    return _ops


def early_starts(record):
    """Number of launches among those of `record()` that may begin before the launch ahead of them has ended: the programmatic
    edges of the graph they are captured into.  Nothing runs."""
    cu = ctypes.CDLL("libcuda.so.1")
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        record()
    raw, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert cu.cuGraphGetEdges_v2(raw, None, None, None, ctypes.byref(n)) == 0
    src, dst, data = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)(), (ctypes.c_ubyte * (8 * n.value))()
    assert cu.cuGraphGetEdges_v2(raw, src, dst, data, ctypes.byref(n)) == 0 and n.value > 0
    return sum(data[8 * i + 2] == 1 for i in range(n.value))       # CUgraphEdgeData::type, programmatic


def layer_args(ops, T, H, I, E, K):
    """Arguments of an inference call of the layer, with buffers of the right sizes and no particular contents."""
    from sonicmoe import _lib
    TK = T * K
    a = _lib.LayerArgs(T, H, I, E, K, TK, -(-TK // 128) * 128 + E * 128)
    u8 = lambda n: torch.zeros(n, dtype=torch.uint8, device=DEV)
    keep = dict(x=u8(2 * T * H), idx=u8(4 * TK), probs=u8(4 * TK), w1=u8(E * 2 * I * H), w1_sf=u8(ops.isa_bytes(E * 2 * I, H)),
                w2=u8(E * H * I), w2_sf=u8(ops.isa_bytes(E * H, I)), out=u8(2 * T * H), counts=u8(4 * E),
                saved=u8(_lib.lib.smoe_layer_bytes(a, 0)), scratch=u8(_lib.lib.smoe_layer_bytes(a, 1)),
                status=ops.status_word(DEV))
    for name, t in keep.items():
        setattr(a, name, t.data_ptr())
    return a, keep


def test_only_the_layer_lets_the_gemms_begin_early(ops):
    """Offsets, counts and weights are read before the kernel ahead has ended where the launch allows it.  In a layer call they
    are complete by then; a caller of the two entry points may have made them with the very kernel ahead."""
    from sonicmoe._lib import check, lib
    T, H, I, E, K = 16, 256, 128, 8, 2
    a, keep = layer_args(ops, T, H, I, E, K)
    st = lambda: torch.cuda.current_stream().cuda_stream
    assert early_starts(lambda: check(lib.smoe_layer_forward(a, st()), "layer")) == 2
    R, P = a.TKp_alloc, lambda t: t.data_ptr()
    i32 = lambda n: torch.zeros(n, dtype=torch.int32, device=DEV)
    md = [i32(n) for n in (E + 1, R, R, T * K, T + 1, R, T * K)]
    ws = torch.zeros(lib.smoe_topk_metadata_workspace(T, E), dtype=torch.uint8, device=DEV)
    xq, y, c = (torch.zeros(n, dtype=torch.uint8, device=DEV) for n in (R * H, R * I, 2 * R * H))
    xsf, ysf = (torch.zeros(ops.isa_bytes(R, n), dtype=torch.uint8, device=DEV) for n in (H, I))

    def metadata_then_gemms():
        check(lib.smoe_topk_metadata(a.idx, a.probs, T, K, E, 128, T * K, R, 0, 0, *map(P, md), a.counts, P(ws), st()), "metadata")
        check(lib.smoe_gemm_gated_few(P(xq), P(xsf), a.w1, a.w1_sf, P(md[0]), a.counts, P(y), P(ysf), R, 2 * I, H, E, a.status,
                                      st()), "gated_few")
        check(lib.smoe_gemm_varlen_m_few(P(y), P(ysf), a.w2, a.w2_sf, P(md[0]), a.counts, P(c), R, H, I, E, a.status, st()),
              "varlen_m_few")

    assert early_starts(metadata_then_gemms) == 0
