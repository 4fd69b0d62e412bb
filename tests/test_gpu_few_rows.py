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


def deq_inputs(shape, g):
    """e4m3 values of N(0,1) and their 1x32 scales, as the quantizers make them."""
    q, sc = Q.row_quant(torch.randn(shape, generator=g).reshape(-1, shape[-1]).to(torch.bfloat16))
    return q.reshape(shape), sc.reshape(*shape[:-1], -1)


def both_forms(ops, counts, H, I, seed, change=None, segments=None):
    """y1 payload, y1 scales and output rows of the live rows from the 256-row kernels and from the few-row ones.  `change` edits
    (x, x scales, w1, w1 scales, w2, w2 scales) of the live rows before; `segments`: rows an expert's segment has, where `counts`
    asks for more."""
    from sonicmoe._lib import check, lib
    g = torch.Generator().manual_seed(seed)
    E = len(counts)
    seg = segments or [-(-c // 128) * 128 for c in counts]
    efo = torch.zeros(E + 1, dtype=torch.int32)
    efo[1:] = torch.cumsum(torch.tensor(seg), 0)
    rows = int(efo[-1]) + 128
    live = torch.cat([torch.arange(int(efo[e]), int(efo[e]) + min(c, seg[e])) for e, c in enumerate(counts)])
    xq = torch.randint(0, 256, (rows, H), generator=g, dtype=torch.uint8)
    xs = torch.randint(0, 256, (rows, H // 32), generator=g, dtype=torch.uint8)
    (lq, ls), (w1, w1s), (w2, w2s) = deq_inputs((len(live), H), g), deq_inputs((E, 2 * I, H), g), deq_inputs((E, H, I), g)
    if change is not None:
        change(lq, ls, w1, w1s, w2, w2s)
    xq[live], xs[live] = lq, ls
    d = lambda t: t.contiguous().to(DEV)
    xq, xsf, w1, w2 = d(xq), d(Q.pack_isa(xs, rows, H)), d(w1), d(w2)
    w1sf = d(Q.pack_isa(w1s.reshape(E * 2 * I, H // 32), E * 2 * I, H))
    w2sf = d(Q.pack_isa(w2s.reshape(E * H, I // 32), E * H, I))
    s_scatter = torch.full((rows,), len(live), dtype=torch.int32)
    s_scatter[live] = torch.arange(len(live), dtype=torch.int32)
    efo, cnt, real, s_scatter = d(efo), *(d(torch.as_tensor(t, dtype=torch.int32)) for t in (counts, [len(live)], s_scatter))
    P, st, status = lambda t: t.data_ptr(), torch.cuda.current_stream().cuda_stream, ops.status_word(DEV).data_ptr()
    out = []
    for few in (False, True):
        y = torch.full((rows, I), 0xAA, dtype=torch.uint8, device=DEV)
        ysf = torch.full((ops.isa_bytes(rows, I),), 0xAA, dtype=torch.uint8, device=DEV)
        c = torch.full((rows, H), 7.0, dtype=torch.bfloat16, device=DEV)
        if few:
            check(lib.smoe_gemm_gated_few(P(xq), P(xsf), P(w1), P(w1sf), P(efo), P(cnt), P(y), P(ysf), rows, 2 * I, H, E, status,
                                          st), "gated_few")
            check(lib.smoe_gemm_varlen_m_few(P(y), P(ysf), P(w2), P(w2sf), P(efo), P(cnt), P(c), rows, H, I, E, status, st),
                  "varlen_m_few")
            dead = torch.ones(rows, dtype=torch.bool)
            dead[live] = False
            assert (y.cpu()[dead] == 0xAA).all() and (c.cpu()[dead] == 7.0).all()            # left as they were
        else:
            check(lib.smoe_gemm_gated_infer(P(xq), P(xsf), P(w1), P(w1sf), P(efo), P(s_scatter), P(real), P(y), P(ysf), rows,
                                            2 * I, H, E, status, st), "gated_infer")
            check(lib.smoe_gemm_varlen_m_live(P(y), P(ysf), P(w2), P(w2sf), P(efo), P(s_scatter), P(real), P(c), rows, H, I, E,
                                              status, st), "varlen_m_live")
        torch.cuda.synchronize()
        ops.check_status(DEV)
        out.append((y.cpu()[live], Q.unpack_isa(ysf.cpu(), rows, I)[live], c.cpu()[live].float()))
    return out


def assert_same_values(a, b):
    """Both forms multiply the same operands; the tensor core may add the products of a K step in another order, which moves a
    value next to a rounding boundary of e4m3 or bf16."""
    (y0, s0, c0), (y1, s1, c1) = a, b
    same = s0 == s1
    assert (~same).float().mean() < 2e-3 and (y0 != y1)[same.repeat_interleave(32, 1)].float().mean() < 2e-3
    assert torch.equal(torch.isnan(c0), torch.isnan(c1)) and torch.equal(torch.isinf(c0), torch.isinf(c1))
    ok = torch.isfinite(c0)
    assert float((c0[ok] - c1[ok]).norm()) <= 4e-3 * float(c0[ok].norm())


def test_nan_and_overflow_leave_the_bytes_of_the_general_kernels(ops):
    """A row of NaN, a NaN in one weight row of an expert, and a row that overflows f32: payload and scale bytes of the up-projection
    included."""
    def change(x, xs, w1, w1s, w2, w2s):
        x[1, 5] = 0x7F                  # every output of row 1
        w1[3, 6, 9] = 0x7F              # one gate column of expert 3, live rows 12 and 13
        xs[4, :] = 0xFE                 # row 4 times 2^127
        x[6] = 0                        # a row of zeros
    a, b = both_forms(ops, [3, 0, 9, 2], 256, 128, 5, change)
    assert_same_values(a, b)
    (y0, s0, c0), (y1, s1, c1) = a, b
    nan = (y0 & 0x7F) == 0x7F
    assert nan[1].all() and nan[12:, 3].all() and not nan[0].any() and torch.equal(nan, (y1 & 0x7F) == 0x7F)
    assert torch.equal(s0[[1, 4, 6]], s1[[1, 4, 6]]) and torch.isnan(c1[[1, 12, 13]]).all() and (c1[6] == 0).all()


@pytest.mark.parametrize("last", [0, 3, 65])
def test_all_256_experts(ops, last):
    counts = [0] * 256
    counts[0], counts[100], counts[254], counts[255] = 1, 17, 2, last
    assert_same_values(*both_forms(ops, counts, 128, 128, 6 + last))


def test_counts_beyond_a_segment_that_was_cut(ops):
    """Metadata made into too small buffers leaves the experts' whole counts beside offsets that are cut."""
    assert_same_values(*both_forms(ops, [140, 70, 500, 9], 256, 128, 7, segments=[128, 128, 256, 0]))


@pytest.mark.parametrize("T,K,E,H,I,few", [
    (40, 8, 8, 256, 128, True), (41, 8, 8, 256, 128, False), (64, 5, 8, 256, 128, True), (64, 6, 8, 256, 128, False),
    (65, 1, 8, 256, 128, True), (80, 1, 8, 256, 128, True), (81, 1, 8, 256, 128, False),             # ten rows on average
    (640, 8, 128, 256, 128, False), (5120, 1, 128, 256, 128, False),                                 # forty
    (192, 1, 64, 6144, 128, True), (193, 1, 64, 6144, 128, False),                                   # one slot: 3 and 4 x 48 tiles
    (128, 4, 64, 6144, 128, True), (129, 4, 64, 6144, 128, False), (128, 5, 64, 128, 3072, False)])  # all slots
def test_which_inference_calls_take_the_few_row_gemms(ops, T, K, E, H, I, few):
    """The few-row GEMMs are the only launches of a layer call that may begin early."""
    from sonicmoe._lib import check, lib
    a, keep = layer_args(ops, T, H, I, E, K)
    n = early_starts(lambda: check(lib.smoe_layer_forward(a, torch.cuda.current_stream().cuda_stream), "layer"))
    assert n == (2 if few else 0)


@pytest.mark.parametrize("T,K,E,busy", [(200, 1, 64, 150), (200, 2, 64, 200), (64, 3, 16, 64), (620, 1, 64, 620)])
def test_inference_with_busy_experts(ops, T, K, E, busy):
    """An expert of up to ten row tiles among idle ones: the output of the training forward, which takes the other kernels."""
    import sonicmoe
    H, I = 256, 128
    g = torch.Generator().manual_seed(T + K)
    logits = torch.rand(T, E, generator=g)
    logits[:busy, 3] = 2.0
    idx = logits.topk(K).indices
    assert not (idx.sort(1).values.diff(dim=1) == 0).any()               # a row's experts are distinct
    idx, scores = idx.to(torch.int32).to(DEV), torch.rand(T, K, generator=g).to(DEV)
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV)
    w1 = (torch.randn(E, 2 * I, H, generator=g) * 0.05).to(torch.bfloat16).to(DEV).requires_grad_(True)
    w2 = (torch.randn(E, H, I, generator=g) * 0.05).to(torch.bfloat16).to(DEV).requires_grad_(True)
    want = sonicmoe.run_sonic_moe(x, idx, scores, K, E, w1, w2, fp8=True).detach()
    with torch.no_grad():
        got = sonicmoe.run_sonic_moe(x, idx, scores, K, E, w1, w2, fp8=True)
    torch.cuda.synchronize()
    ops.check_status(DEV)
    assert float((got.float() - want.float()).norm()) <= 4e-3 * float(want.float().norm())
