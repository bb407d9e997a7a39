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
    if not events:
        pytest.skip("the profiler sees no kernels here (another tool may hold it)")
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


@pytest.mark.parametrize("B,H,KV,hd,positions,chunks", [(1, 8, 2, 128, 8192, True), (2, 4, 1, 256, 4096, True), (1, 12, 3, 64, 40, True), (1, 3, 3, 64, 40, False), (64, 16, 2, 64, 300, False),
                                                        (16, 8, 2, 128, 300, False)])
def test_attention_of_a_step_long_caches_in_chunks(dev, B, H, KV, hd, positions, chunks):
    """Few key heads over a long cache need more CTAs than a cluster has; many sequences, whose warps work alone, do not."""
    m = llama(dev, H=H, KV=KV, hd=hd, positions=16384)
    m.cache_reserve(B, positions)
    m.forward_cached(np.zeros((B, 1), np.int32), want_logits=False)
    names = kernels(dev, lambda: m.decode_step(B))
    assert any("attention_chunk_kernel" in n for n in names) == chunks and any("attention_kernel" in n for n in names) != chunks, names


@pytest.mark.parametrize("B,H,KV,hd", [(1, 8, 2, 128), (3, 8, 1, 64), (1, 2, 2, 256), (2, 3, 1, 80)])
def test_steps_over_a_long_capacity_repeat_those_over_a_short_one(dev, B, H, KV, hd):
    """The same tokens through the two attention kernels of a step (the capacity decides), and after growing from one to the other."""
    ids = np.random.default_rng(hd).integers(0, 500, (B, 90)).astype(np.int32)
    out = []
    for reserve in (0, 16000):
        m = llama(dev, H=H, KV=KV, hd=hd, positions=16384, L=2)
        if reserve:
            m.cache_reserve(B, reserve)
        out.append([m.forward_cached(ids[:, :40])] + [m.forward_cached(ids[:, t:t + 1]) for t in range(40, 80)] + [m.forward_cached(ids[:, 80:83])])
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 1e-5 * np.abs(a).max()


def test_the_tensor_cores_can_be_turned_off_for_prompts(monkeypatch):
    monkeypatch.setenv("RUAI_B200_TC", "0")
    dev = nn.Device(0)
    m = llama(dev)
    names = kernels(dev, lambda: prompt(m, np.zeros((1, 200), np.int32)))
    assert any("attention_prefill_kernel" in n for n in names) and not any("_tc" in n for n in names), names
    m.close()


@pytest.mark.parametrize("bits,k,n,tc", [(8, 2048, 2048, False), (8, 1024, 19456, True), (8, 4096, 5120, True), (4, 4096, 4096, False), (4, 14336, 4096, False)])
def test_one_row_by_itself_runs_on_the_shorter_kernel(dev, bits, k, n, tc):
    if bits == 8:
        w = nn.QWeight.int8(dev, np.ones((k, n), np.int8), np.ones(n, np.float32))
    else:
        w = nn.QWeight.int4(dev, np.full((k // 2, n), 0x11, np.int8), np.ones((k // 32, n), np.float32), 32)
    x = nn.Tensor.from_numpy(dev, np.ones((1, k), np.float32))
    names = kernels(dev, lambda: nn._matmul_q(x, w))
    assert any("gemv_tc" in name for name in names) == tc and any("row_kernel" in name for name in names) != tc, names
    assert np.array_equal(nn._matmul_q(x, w).numpy(), np.full((1, n), float(k), np.float32))
