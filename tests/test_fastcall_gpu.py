"""The native form of the plain calls (csrc/fastcall.cpp) against the general form of ops.py, which takes over where a stream
is named: the same bits, the same refusals."""
import concurrent.futures

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from inference_b200 import ops as _ops
    assert _ops.has_cuda() and _ops.device_sm_version(0) == 100, "needs a B200"
    return _ops


def calls(ops, dt):
    """name -> function of the keyword arguments that force a form"""
    from inference_b200 import synth
    g = torch.Generator(device="cuda").manual_seed(3)
    x = synth.activations(33, 512, seed=1).to(dt)
    res = torch.randn((33, 512), device="cuda", generator=g).to(dt)
    w = torch.randn(512, device="cuda", generator=g).to(dt)
    bq, bs = synth.quantised_weights(200, 512, seed=2)
    q, s = ops.quant_fp8_per_token_group(x)
    heads = torch.randn((33, 4, 64), device="cuda", generator=g).to(dt)
    pos = torch.arange(33, device="cuda")
    cache = torch.randn((2, 40, 16, 2, 64), device="cuda", generator=g).to(dt)
    tables = torch.arange(33, device="cuda", dtype=torch.int32).view(33, 1)
    lens = torch.full((33,), 11, device="cuda", dtype=torch.int32)

    def add_norm(**k):
        r = res.clone()
        return (*ops.rmsnorm_quant(x, w, residual=r, **k), r)
    return {
        "quant": lambda **k: ops.quant_fp8_per_token_group(x, **k),
        "gemm": lambda **k: (ops.w8a8_block_fp8_gemm(q, s, bq, bs, torch.float32, **k),),
        "fused": lambda **k: (ops.w8a8_block_fp8_gemm_fused_quant(x, bq, bs, dt, **k),),
        "norm": lambda **k: ops.rmsnorm_quant(x, w, 1e-5, **k),
        "add_norm": add_norm,
        "rope": lambda **k: (ops.rope_neox(heads.clone(), pos, 32, 500000, 0.5, **k),),
        "attn": lambda **k: (ops.paged_attn_decode(heads, cache[0], cache[1], tables, lens, 0.125, **k),),
    }


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("name", ["quant", "gemm", "fused", "norm", "add_norm", "rope", "attn"])
def test_both_forms_agree(ops, dt, name):
    call = calls(ops, dt)[name]
    for a, b in zip(call(), call(stream=torch.cuda.current_stream()), strict=True):
        assert a.dtype == b.dtype and a.shape == b.shape and a.is_contiguous() and torch.equal(a, b)
    side = torch.cuda.Stream()      # the current stream is the one that is used
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        c = call()
    side.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(call(), c))


def test_what_is_not_plain_goes_the_general_way(ops):
    from inference_b200 import _capi
    x = torch.randn((4, 256), device="cuda", dtype=torch.bfloat16)
    q, s = ops.quant_fp8_per_token_group(x)

    class Sub(torch.Tensor):
        pass
    fast = _capi.fast
    assert fast.quant(x.cpu()) is None and fast.quant(x.t()) is None and fast.quant(x[0]) is None
    assert fast.quant(x.double()) is None and fast.quant(x[:, :100].contiguous()) is None and fast.quant(None) is None
    assert fast.quant(x.as_subclass(Sub)) is None
    assert all(torch.equal(a, b) for a, b in zip(ops.quant_fp8_per_token_group(x.as_subclass(Sub)), (q, s)))
    for bad, error in ((x.cpu(), ValueError), (x.t(), ValueError), (x.double(), ValueError), (x[:, :100].contiguous(), ops.InferopError),
                       (x[:0], ops.InferopError)):
        with pytest.raises(error):
            ops.quant_fp8_per_token_group(bad)
    with pytest.raises(KeyError):
        ops.w8a8_block_fp8_gemm(q, s, q, torch.ones((1, 2), device="cuda"), torch.float64)
    with pytest.raises(ValueError):
        ops.w8a8_block_fp8_gemm(q, s, q, torch.ones((2, 2), device="cuda"))
    with pytest.raises(ops.InferopError):       # the C ABI's own refusal (b_q not 16-byte aligned) by the native form
        flat = torch.zeros(256 * 128 + 1, device="cuda", dtype=torch.uint8)
        ops.w8a8_block_fp8_gemm(q, s, flat[1:].view(128, 256), torch.ones((1, 2), device="cuda"))


def test_several_threads(ops):
    call = calls(ops, torch.bfloat16)
    want = {n: f() for n, f in call.items()}
    torch.cuda.synchronize()

    def work():
        done = 0
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(50):
                for n, f in call.items():
                    assert all(torch.equal(a, b) for a, b in zip(f(), want[n])), n
                done += 1
        return done
    with concurrent.futures.ThreadPoolExecutor(4) as pool:
        runs = [pool.submit(work) for _ in range(4)]
        assert [r.result() for r in runs] == [50] * 4      # (what a thread raised is raised here)
