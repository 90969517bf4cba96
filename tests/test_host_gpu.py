"""The host-buffer front end gives the same bits as the device-pointer operators."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_host_linear_equals_device_path():
    from inference_b200 import ops, synth
    from inference_b200.host import HostLinearFP8
    m, n, k = 1000, 640, 1024   # several panels, the last one ragged
    x = synth.activations(m, k, seed=4)
    bq, bs = synth.quantised_weights(n, k, seed=4)
    aq, a_s = ops.quant_fp8_per_token_group(x)
    want = ops.w8a8_block_fp8_gemm(aq, a_s, bq, bs, torch.bfloat16).cpu()
    lin = HostLinearFP8(bq, bs, max_rows=m, panel_rows=256)
    x_host = x.cpu().pin_memory()
    out = torch.empty((m, n), dtype=torch.bfloat16).pin_memory()
    for _ in range(2):   # buffers are reused across calls
        out.fill_(0)
        lin(x_host, out)
        assert torch.equal(out.view(torch.int16), want.view(torch.int16))
    assert ops.device_status()[0] == 0


@pytest.mark.parametrize("m,panel_rows", [(1000, 256), (1000, 240), (100, 48), (65, 64), (64, 20), (300, 1000)])
def test_the_bits_do_not_depend_on_the_panels(m, panel_rows):
    """Panels, or a last panel, of so few rows that a call of their own would be cut along K; unrounded results."""
    from inference_b200 import ops, synth
    from inference_b200.host import HostLinearFP8
    n, k = 640, 1024
    x = synth.activations(m, k, seed=m)
    bq, bs = synth.quantised_weights(n, k, seed=4)
    aq, a_s = ops.quant_fp8_per_token_group(x)
    want = ops.w8a8_block_fp8_gemm(aq, a_s, bq, bs, torch.float32).cpu()
    lin = HostLinearFP8(bq, bs, max_rows=max(m, 300), panel_rows=panel_rows, out_dtype=torch.float32)
    x_host, out = x.cpu().pin_memory(), torch.zeros((m, n)).pin_memory()
    for _ in range(2):
        out.fill_(0)
        assert torch.equal(lin(x_host, out), want)
