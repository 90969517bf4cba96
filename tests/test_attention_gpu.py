"""Paged attention decode through the C ABI against the oracle (reference/reference.cpp:112-150) with
the cases and tolerances of the reference's own GPU test (tests/test_paged_attn.cpp:110-117) and more:
shuffled physical blocks, empty sequences, groups of 1 / 2 / 4 / 8 query heads per KV head, sequences
long enough to be cut into several token ranges."""
import time

import numpy as np
import pytest
import torch

import oracle
from test_oracle_cpu import attn_case

pytestmark = pytest.mark.gpu

TOL = {torch.float32: (2e-3, 2e-3), torch.float16: (5e-3, 5e-3), torch.bfloat16: (2e-2, 2e-2)}


@pytest.fixture(scope="module")
def ops():
    from inference_b200 import ops as _ops
    assert _ops.has_cuda() and _ops.device_sm_version(0) == 100, "needs a B200"
    return _ops


@pytest.fixture(autouse=True, params=[0, 1, 2], ids=["auto", "cuda_cores", "tensor_cores"])
def form(request, ops):
    """16-bit caches are served in two forms, chosen by size: every test here runs with the choice and with either."""
    ops.set_option("attn_path", request.param)
    yield request.param
    ops.set_option("attn_path", 0)


def rounded(a, dtype):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dtype).float().numpy()


def run_case(ops, dtype, batch, heads, kv_heads, dim, block_size, lens, shuffle, seed=0):
    q, k, v, tables, sl = attn_case(batch, heads, kv_heads, dim, block_size, lens, seed=seed, shuffle=shuffle)
    q, k, v = rounded(q, dtype), rounded(k, dtype), rounded(v, dtype)
    scale = float(1.0 / np.sqrt(dim))
    want = oracle.paged_attn_decode(q, k, v, tables, sl, scale)
    cu = lambda a, dt=None: torch.from_numpy(a).cuda().to(dt) if dt is not None else torch.from_numpy(a).cuda()
    got = ops.paged_attn_decode(cu(q, dtype), cu(k, dtype), cu(v, dtype), cu(tables), cu(sl), scale)
    torch.cuda.synchronize()
    return got.float().cpu().numpy(), want


@pytest.mark.parametrize("case,dtype", [
    ((3, 32, 8, 128, 16, [1, 17, 129]), torch.float32),
    ((3, 32, 8, 128, 16, [1, 17, 129]), torch.bfloat16),
    ((2, 16, 4, 64, 16, [5, 64]), torch.bfloat16),
    ((2, 8, 8, 256, 16, [33, 200]), torch.bfloat16),
    ((1, 32, 8, 128, 16, [2048]), torch.bfloat16),
])
def test_the_reference_tests_own_cases(ops, case, dtype):
    got, want = run_case(ops, dtype, *case, shuffle=False)
    rtol, atol = TOL[dtype]
    np.testing.assert_allclose(got, want, rtol=rtol, atol=atol)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("heads,kv_heads", [(8, 8), (8, 4), (16, 4), (32, 4), (6, 2), (5, 5), (12, 4)])
@pytest.mark.parametrize("dim", [64, 128, 256])
def test_head_groups_and_head_sizes(ops, dtype, heads, kv_heads, dim):
    got, want = run_case(ops, dtype, 3, heads, kv_heads, dim, 16, [1, 40, 333], shuffle=True, seed=heads + dim)
    rtol, atol = TOL[dtype]
    np.testing.assert_allclose(got, want, rtol=rtol, atol=atol)
    if dtype == torch.float32:
        np.testing.assert_allclose(got, want, rtol=2e-5, atol=2e-5)   # far inside the reference's 2e-3


@pytest.mark.parametrize("block_size", [1, 8, 16, 32, 128])
def test_block_sizes_empty_sequences_and_long_ones(ops, block_size):
    lens = [0, 1, 4097, 0, 777, 9000]
    got, want = run_case(ops, torch.bfloat16, len(lens), 8, 2, 128, block_size, lens, shuffle=True, seed=block_size)
    np.testing.assert_allclose(got, want, rtol=2e-2, atol=2e-2)
    assert np.array_equal(got[0], np.zeros_like(got[0])) and np.array_equal(got[3], np.zeros_like(got[3]))


def test_a_single_long_sequence_is_cut_into_ranges_and_merged(ops):
    got, want = run_case(ops, torch.float32, 1, 16, 2, 128, 16, [20000], shuffle=True, seed=9)
    np.testing.assert_allclose(got, want, rtol=5e-5, atol=5e-5)
    # sequence lengths beyond the table are clamped to what the table covers
    q, k, v, tables, sl = attn_case(2, 4, 2, 64, 16, [48, 48], seed=3)
    scale = 0.125
    want = oracle.paged_attn_decode(q, k, v, tables, sl, scale)
    big = np.array([1000, 48], np.int32)
    cu = lambda a: torch.from_numpy(a).cuda()
    got = ops.paged_attn_decode(cu(q), cu(k), cu(v), cu(tables), cu(big), scale).cpu().numpy()
    np.testing.assert_allclose(got, want, rtol=2e-5, atol=2e-5)


def test_length_one_returns_the_value_row_and_outputs_stay_in_range(ops):
    q, k, v, tables, sl = attn_case(3, 32, 8, 128, 16, [1, 17, 129])
    cu = lambda a: torch.from_numpy(a).cuda()
    out = ops.paged_attn_decode(cu(q), cu(k), cu(v), cu(tables), cu(sl), float(1 / np.sqrt(128))).cpu().numpy()
    np.testing.assert_allclose(out[0, 0], v[tables[0, 0], 0, 0], atol=1e-5)
    assert out.min() >= v.min() - 1e-3 and out.max() <= v.max() + 1e-3


def test_rejected_calls(ops):
    from inference_b200 import _capi
    lib = _capi.lib
    t = torch.zeros(1 << 14, dtype=torch.float32, device="cuda")
    p = t.data_ptr()
    i = torch.zeros(16, dtype=torch.int32, device="cuda").data_ptr()
    assert lib.inferop_paged_attn_decode(p, p, p, p, i, i, 0, 1, 8, 3, 128, 16, 4, 0.1, None) == _capi.ERR_SHAPE    # 8 % 3
    assert lib.inferop_paged_attn_decode(p, p, p, p, i, i, 0, 1, 8, 4, 96, 16, 4, 0.1, None) == _capi.ERR_SHAPE     # head_dim
    assert lib.inferop_paged_attn_decode(p, p, p, p, i, i, 4, 1, 8, 4, 128, 16, 4, 0.1, None) == _capi.ERR_DTYPE
    assert lib.inferop_paged_attn_decode(p, p, p + 4, p, i, i, 0, 1, 8, 4, 128, 16, 4, 0.1, None) == _capi.ERR_POINTER
    assert lib.inferop_paged_attn_decode(p, p, p, p, None, i, 0, 1, 8, 4, 128, 16, 4, 0.1, None) == _capi.ERR_POINTER
    torch.cuda.synchronize()
    assert bool((t == 0).all())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("heads,kv_heads,dim,block_size,lens", [
    (7, 1, 128, 16, [15, 16, 17, 63, 64, 65]),                  # edges of a warp's block and of a unit; 7 rows
    (9, 1, 64, 16, [127, 128, 129, 1, 0, 200]),                 # 9 query heads of a KV head: three CTAs of three
    (24, 2, 64, 3, [1, 2, 3, 4, 191, 192, 193]),                # 12 of a KV head (two CTAs of six), odd block size
    (8, 8, 256, 16, [65, 64, 5]),
    (4, 1, 64, 64, [int(x) for x in range(0, 300, 7)]),         # more sequences than a warp has lanes
    (16, 2, 128, 16, [30000, 1, 64 * 40]),                      # a pair spread over many CTAs beside short ones
])
def test_16_bit_caches_at_the_edges_of_units_and_heads(ops, dtype, heads, kv_heads, dim, block_size, lens):
    got, want = run_case(ops, dtype, len(lens), heads, kv_heads, dim, block_size, lens, shuffle=True, seed=len(lens))
    # one rounding of the output, and probabilities of at least 22 bits: 1e-4 is twenty times their effect
    rtol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -10
    np.testing.assert_allclose(got, want, rtol=rtol, atol=1e-4)


def test_16_bit_caches_large_batches_and_unaligned_queries(ops):
    lens = [(i * 37) % 90 for i in range(1030)]   # more sequences than the evenly cut form takes
    got, want = run_case(ops, torch.bfloat16, len(lens), 2, 1, 64, 16, lens, shuffle=True, seed=4)
    np.testing.assert_allclose(got, want, rtol=2.0 ** -8, atol=1e-4)
    q, k, v, tables, sl = attn_case(2, 4, 2, 64, 16, [40, 70], seed=3)
    cu = lambda a, dt: torch.from_numpy(a).cuda().to(dt)
    buf = torch.zeros(q.size + 1, dtype=torch.bfloat16, device="cuda")
    buf[1:] = cu(q, torch.bfloat16).reshape(-1)
    args = cu(k, torch.bfloat16), cu(v, torch.bfloat16), torch.from_numpy(tables).cuda(), torch.from_numpy(sl).cuda(), 0.125
    a = ops.paged_attn_decode(buf[1:].view(q.shape), *args)
    b = ops.paged_attn_decode(buf[1:].view(q.shape).clone(), *args)
    assert torch.equal(a, b)


def long_case(ops, seed, lens=(20000, 7000, 13111)):
    q, k, v, tables, sl = attn_case(len(lens), 32, 8, 64, 16, list(lens), seed=seed)
    args = [torch.from_numpy(a).cuda().to(torch.float16) for a in (q, k, v)]
    args += [torch.from_numpy(tables).cuda(), torch.from_numpy(sl).cuda(), 0.125]
    want = ops.paged_attn_decode(*args)
    torch.cuda.synchronize()
    return args, want


def test_16_bit_caches_captured_on_a_stream_without_scratch(ops):
    """A stream's first call may be inside a graph capture: the graph gets scratch of its own and the evenly cut form,
    bit for bit what the call gives outside."""
    args, want = long_case(ops, 6)
    out = torch.zeros_like(want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        ops.paged_attn_decode(*args, out=out)
    for _ in range(2):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)


def test_a_captured_call_shares_no_scratch_with_its_streams_other_calls(ops):
    (args1, want1), (args2, want2) = long_case(ops, 10), long_case(ops, 11, (9001, 16000))
    out1, out2 = torch.zeros_like(want1), torch.zeros_like(want2)
    a, b, c = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Stream()
    outs = [torch.zeros_like(want1) for _ in range(2)]
    ops.paged_attn_decode(*args2, out=out2, stream=a)
    torch.cuda.synchronize()
    graphs = [torch.cuda.CUDAGraph() for _ in range(2)]
    for graph, out in zip(graphs, outs):
        with torch.cuda.graph(graph, stream=a):
            for _ in range(3):
                ops.paged_attn_decode(*args1, out=out)
    for _ in range(40):   # the graphs and the stream they were captured on, all at once
        for graph, stream in zip(graphs, (b, c)):
            with torch.cuda.stream(stream):
                graph.replay()
        for _ in range(3):
            ops.paged_attn_decode(*args2, out=out2, stream=a)
        torch.cuda.synchronize()
        assert torch.equal(outs[0], want1) and torch.equal(outs[1], want1) and torch.equal(out2, want2)
        for t in (*outs, out2):
            t.zero_()
        torch.cuda.synchronize()


def test_scratch_of_a_graph_is_given_back_with_it(ops):
    """More captures than there are sets, one after the other, and more calls than a set's counters last for."""
    args, want = long_case(ops, 6)
    for i in range(80):
        out = torch.zeros_like(want)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(1 if i else 150):
                ops.paged_attn_decode(*args, out=out)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want), i
        del graph
    for _ in range(150):
        out = ops.paged_attn_decode(*args)
    assert torch.equal(out, want)


def test_captures_beyond_the_scratch_sets_still_run(ops):
    """256 graphs hold every set: further captures take a form that needs none, until graphs are destroyed."""
    args, want = long_case(ops, 6)
    graphs, out = [], torch.zeros_like(want)

    def capture():
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            ops.paged_attn_decode(*args, out=out)
        return graph

    def replay(graph):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        return out

    for _ in range(258):
        graphs.append(capture())
    assert torch.equal(replay(graphs[0]), want) and torch.equal(replay(graphs[100]), want)
    got = replay(graphs[257])
    assert not torch.equal(got, want)   # (another order of sums)
    # both are rounded once to fp16, from sums that differ by fp32's rounding
    torch.testing.assert_close(got, want, rtol=2.0 ** -10, atol=1e-6)
    graphs.clear()
    torch.cuda.synchronize()
    time.sleep(0.2)   # the sets come back on a thread of the driver's
    assert torch.equal(replay(capture()), want)


def place(tables, block_size, b, t):
    """Where token t of sequence b lies in the cache: (block, offset)."""
    return tables[b, t // block_size], t % block_size


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("dim", [64, 128, 256])
def test_infinities_and_nan_in_the_value_cache(ops, dtype, dim):
    """p * inf is inf for every p > 0, in a sequence of one CTA and in one that several share."""
    q, k, v, tables, sl = attn_case(3, 8, 2, dim, 16, [40, 5000, 1], seed=5, shuffle=True)
    q, k, v = rounded(q, dtype), rounded(k, dtype), rounded(v, dtype)
    for b, t, h, d, val in [(0, 20, 0, 5, np.inf), (0, 39, 1, 7, -np.inf), (1, 4999, 0, 0, np.inf), (1, 70, 0, dim - 1, -np.inf),
                            (1, 3000, 1, 9, np.inf), (1, 17, 1, 9, -np.inf), (2, 0, 1, 3, np.inf), (1, 100, 0, 50, np.nan)]:
        blk, off = place(tables, 16, b, t)
        v[blk, off, h, d] = val
    scale = float(1 / np.sqrt(dim))
    want = oracle.paged_attn_decode(q, k, v, tables, sl, scale)
    assert np.isinf(want).sum() == 4 * 7 and np.isnan(want).sum() == 4 * 2   # (the first block is every sequence's)
    cu = lambda a, dt: torch.from_numpy(a).cuda().to(dt)
    got = ops.paged_attn_decode(cu(q, dtype), cu(k, dtype), cu(v, dtype), torch.from_numpy(tables).cuda(),
                                torch.from_numpy(sl).cuda(), scale).float().cpu().numpy()
    rtol, atol = TOL[dtype]
    np.testing.assert_allclose(got, want, rtol=rtol, atol=atol)   # (NaN where the oracle has NaN, infinities of its sign)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("gap", [14.0, 17.5, 24.0, 25.01, 28.0])
def test_small_probabilities_stay_in_the_sum(ops, dtype, gap):
    """One key scores `gap` powers of two above 4095 equal ones and has V = 0, the others V = 1: the output is
    their share of the denominator.  300 sequences, so that one warp sees the large score and many small ones."""
    batch, heads, n = 300, 8, 4096
    q = np.zeros((batch, heads, 64), np.float32)
    q[:, :, 0] = 8
    k = np.zeros((n // 16, 16, 1, 64), np.float32)
    v = np.ones_like(k)
    k[0, 1, 0, 0] = gap * np.log(2)
    v[0, 1] = 0
    k = rounded(k, dtype)
    tail = (n - 1) * np.exp(-np.float64(k[0, 1, 0, 0]))
    want = tail / (1 + tail)
    cu = lambda a, dt: torch.from_numpy(a).cuda().to(dt)
    tables = torch.arange(n // 16, dtype=torch.int32, device="cuda").repeat(batch, 1)
    got = ops.paged_attn_decode(cu(q, dtype), cu(k, dtype), cu(v, dtype), tables,
                                torch.full((batch,), n, dtype=torch.int32, device="cuda"), 0.125).double().cpu().numpy()
    # one rounding of the output (11, 8 or 24 bits; half of fp16's smallest step at its low end); a score of up
    # to 28 in fp32 and the 2-ulp exponential: 28 x 2^-24 + 2^-22 in the share, and as much again for the sums
    unit = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8, torch.float32: 2.0 ** -24}[dtype]
    floor = 2.0 ** -25 if dtype == torch.float16 else 0.0
    np.testing.assert_allclose(got, want, rtol=unit + 2 * (28 * 2.0 ** -24 + 2.0 ** -22), atol=floor)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("dim", [64, 128, 256])
def test_keys_that_score_minus_infinity(ops, dtype, dim):
    """A block, a warp's range or a CTA's range of such keys has no weight; a sequence of nothing else has no answer."""
    q, k, v, tables, sl = attn_case(3, 8, 2, dim, 16, [400, 9000, 40], seed=8, shuffle=True)
    q[:, :, 3] = np.abs(q[:, :, 3]) + 0.1
    q[0, 5, 3] = -1    # this head's scores are +inf there
    q, k, v = rounded(q, dtype), rounded(k, dtype), rounded(v, dtype)
    for b, t0, t1 in ((0, 0, 48), (0, 60, 61), (1, 16, 1000), (1, 3000, 3300), (2, 16, 40)):   # (the first block is every sequence's)
        for t in range(t0, t1):
            blk, off = place(tables, 16, b, t)
            k[blk, off, :, 3] = -np.inf
    scale = float(1 / np.sqrt(dim))
    want = oracle.paged_attn_decode(q, k, v, tables, sl, scale)
    assert np.isnan(want[0]).sum() == dim and not np.isnan(want[1]).any() and np.isnan(want[2]).all()
    cu = lambda a, dt: torch.from_numpy(a).cuda().to(dt)
    got = ops.paged_attn_decode(cu(q, dtype), cu(k, dtype), cu(v, dtype), torch.from_numpy(tables).cuda(),
                                torch.from_numpy(sl).cuda(), scale).float().cpu().numpy()
    rtol, atol = TOL[dtype]
    np.testing.assert_allclose(got, want, rtol=rtol, atol=atol)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_what_lies_behind_a_sequence_is_not_read_into_it(ops, dtype):
    """NaN in every cache row that is no token's: in the rest of a last block, in unused blocks."""
    q, k, v, tables, sl = attn_case(4, 8, 2, 128, 16, [40, 5000, 1, 0], seed=6, shuffle=True)
    q, k, v = rounded(q, dtype), rounded(k, dtype), rounded(v, dtype)
    want = oracle.paged_attn_decode(q, k, v, tables, sl, 0.0884)
    used = np.zeros(k.shape[:2], bool)
    for b in range(4):
        for t in range(sl[b]):
            used[place(tables, 16, b, t)] = True
    k[~used] = np.nan
    v[~used] = np.nan
    cu = lambda a, dt: torch.from_numpy(a).cuda().to(dt)
    got = ops.paged_attn_decode(cu(q, dtype), cu(k, dtype), cu(v, dtype), torch.from_numpy(tables).cuda(),
                                torch.from_numpy(sl).cuda(), 0.0884).float().cpu().numpy()
    rtol, atol = TOL[dtype]
    np.testing.assert_allclose(got, want, rtol=rtol, atol=atol)


def test_a_streams_first_call_leaves_another_streams_capture_alone(ops):
    q, k, v, tables, sl = attn_case(80, 32, 8, 64, 16, [33] * 80, seed=7)
    args = [torch.from_numpy(a).cuda().to(torch.bfloat16) for a in (q, k, v)]
    args += [torch.from_numpy(tables).cuda(), torch.from_numpy(sl).cuda(), 0.125]
    want = ops.paged_attn_decode(*args)
    captured, eager, fresh = torch.zeros_like(want), torch.zeros_like(want), torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured.copy_(want)
        ops.paged_attn_decode(*args, out=eager, stream=fresh)   # its scratch is allocated here
        captured.add_(1)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(eager, want) and torch.equal(captured, want + 1)


@pytest.mark.parametrize("dim", [64, 128, 256])
@pytest.mark.parametrize("heads,length", [(8, 130), (8, 20000), (5, 3000), (4, 40000)])
def test_one_pair_shared_by_a_few_or_many_ctas(ops, dim, heads, length):
    """All heads on one KV head, one sequence: 3 to 53 parts to merge, full and partial batches of them."""
    got, want = run_case(ops, torch.float16, 1, heads, 1, dim, 16, [length], shuffle=True, seed=length)
    np.testing.assert_allclose(got, want, rtol=2.0 ** -10, atol=1e-4)


def test_options_of_the_cuda_core_form_select_it(ops, form):
    args, _ = long_case(ops, 12)   # (tensor cores of themselves)
    try:
        for key, value in (("attn_splits", 1), ("attn_splits", 5), ("attn_heads_per_cta", 2)):
            ops.set_option(key, value)
            got = ops.paged_attn_decode(*args)
            ops.set_option("attn_path", 1)
            want = ops.paged_attn_decode(*args)
            ops.set_option("attn_path", form)
            assert torch.equal(got, want) == (form != 2)
            ops.set_option(key, 0)
    finally:
        ops.set_option("attn_splits", 0)
        ops.set_option("attn_heads_per_cta", 0)
    if form == 0:
        got = ops.paged_attn_decode(*args)
        assert not torch.equal(got, want)
        ops.set_option("attn_path", 2)
        assert torch.equal(got, ops.paged_attn_decode(*args))


@pytest.mark.parametrize("batch,length,heads,kv_heads,dim", [(3, 20000, 32, 8, 128), (64, 777, 32, 8, 64), (2, 20000, 8, 8, 128),
                                                             (2, 9000, 16, 4, 256)])
def test_long_sums_are_as_good_as_fp32_additions(ops, batch, length, heads, kv_heads, dim):
    """V around 1: a sum that is off by e, always to the same side or not, is rounded to another fp16 value in e / 2^-10 of
    the elements.  Eight roundings of 2^-24 make 2^-11 of them; the bound is twice that."""
    g = torch.Generator(device="cuda")
    g.manual_seed(length)
    per = -(-length // 16)
    rand = lambda *shape: torch.randn(shape, device="cuda", generator=g)
    q = (2 * rand(batch, heads, dim)).half()
    k = rand(batch * per, 16, kv_heads, dim).half()
    v = (rand(batch * per, 16, kv_heads, dim).half() + 1).half()
    tables = torch.randperm(batch * per, device="cuda", generator=g).to(torch.int32).view(batch, per)
    scale = dim ** -0.5
    got = ops.paged_attn_decode(q, k, v, tables, torch.full((batch,), length, dtype=torch.int32, device="cuda"), scale)
    wrong = 0
    for b in range(batch):
        kk, vv = (c[tables[b].long()].reshape(-1, kv_heads, dim)[:length].double() for c in (k, v))
        p = torch.softmax(torch.einsum("kgd,tkd->kgt", q[b].double().view(kv_heads, -1, dim), kk) * scale, -1)
        wrong += int((got[b] != torch.einsum("kgt,tkd->kgd", p, vv).reshape(heads, dim).half()).sum())
    assert wrong <= got.numel() * 2.0 ** -10
