"""Which kernels a call runs, where that is part of what it promises."""
import numpy as np
import pytest

import zazasun_cases as zcases
from ruai_b200 import nn

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert nn.Device.is_available(), "these tests need a CUDA device"
    return nn.Device.cuda(0)


def kernels(dev, call):
    """Names of the kernels that `call` launches, in order."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.init()
    call()  # allocations and attributes
    dev.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        dev.synchronize()
        torch.cuda.synchronize()
    events = [e for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    return [e.name for e in sorted(events, key=lambda e: e.time_range.start)]


def llama(dev, H=8, KV=2, hd=64, V=500, d=256, ff=512, L=1, bits=8, positions=4096):
    m = nn.Llama(dev, nn.LlamaConfig(V, d, ff, L, H, KV, hd, positions, 1e-5, 10000.0, 0))
    m.load_synthetic(5, bits, 32)
    return m


def prompt(m, ids):
    m.cache_clear()
    m.forward_cached(ids, want_logits=False)


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_layer_list_decoders_keep_f32_attention(dev, dtype):
    """Their roundings of every layer's output follow the order of the sums: a prompt's attention is the f32 kernel at every length."""
    cfg = zcases.config([zcases.attention(), zcases.attention(heads=3, kv_heads=1, dim=12, vdim=12, size=17, keep_first=1)])
    m = nn.Zazasun(dev, nn.ZazasunConfig(cfg, 0))
    for name, t in zcases.weights(cfg).items():
        m.set_tensor(name, t)
    m.build(dtype)
    for T in (95, 96, 200):
        names = kernels(dev, lambda: prompt(m, zcases.tokens(cfg, T)[None]))
        assert sum("attention_prefill_kernel" in n for n in names) == 2 and not any("attn_tc_kernel" in n for n in names), (T, names)


def test_long_prompts_of_quantized_decoders_use_the_tensor_cores(dev):
    m = llama(dev)
    for T, tc in ((95, False), (96, True), (300, True)):
        names = kernels(dev, lambda: prompt(m, np.zeros((1, T), np.int32)))
        assert any("attn_tc_kernel" in n for n in names) == tc and any("attention_prefill_kernel" in n for n in names) != tc, (T, names)
