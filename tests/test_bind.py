"""The CPython binding behind the operators: what is refused before anything is launched (CPU), and on the GPU that a call lands on the current stream of
its tensors' device, takes whatever int() takes, and shares the work spaces that the Python functions hand out."""
import threading

import pytest
import torch

HALF = torch.half


def test_refusals_before_a_launch():
    from qserve_b200 import backend as b

    x, w, o = torch.zeros(2, 128, dtype=torch.int8), torch.zeros(128, 64, dtype=torch.int8), torch.zeros(2, 128, dtype=HALF)
    s = torch.ones(128, dtype=HALF)
    with pytest.raises(RuntimeError, match="in_feats must be on CUDA"):
        b.w4a8_per_chn_gemm_forward_cuda(x, w, s, s, s, s, o)
    with pytest.raises(TypeError):
        b.w4a8_per_chn_gemm_forward_cuda(None, w, s, s, s, s, o)
    with pytest.raises(TypeError):
        b.invoke_quant_fuse_sum(x, o, None, s)
    with pytest.raises(RuntimeError, match="input must be on CUDA"):
        b.silu_and_mul(o, o)
    with pytest.raises(RuntimeError, match="q must be on CUDA"):
        b.single_query_attention(o, o, o, o, None, None, 8192, 64, 64, 1, 128, 1e4, True, True, True)


@pytest.mark.gpu
def test_streams_threads_and_integers(dev):
    from qserve_b200 import backend as b

    g = torch.Generator(device=dev).manual_seed(0)
    M, N, K = 33, 256, 512
    x = torch.randint(-127, 128, (M, K), dtype=torch.int8, device=dev, generator=g)
    w = torch.randint(-127, 128, (N, K), dtype=torch.int8, device=dev, generator=g)
    s, a = torch.rand(N, device=dev).half() * 0.01, torch.rand(M, device=dev).half() * 0.01
    want = ((x.double() @ w.double().t()) * (s.float()[None] * a.float()[:, None]).double()).half()
    outs = [torch.zeros(M, N, dtype=HALF, device=dev) for _ in range(4)]

    def work(i):
        st = torch.cuda.Stream(dev)
        st.wait_stream(torch.cuda.default_stream(dev))
        with torch.cuda.stream(st):
            for _ in range(20):
                b.w8a8_gemm_forward_cuda(x, w, s, a, outs[i])
        st.synchronize()

    torch.cuda.synchronize()
    for i in range(4):  # one thread at a time: the split-K work space belongs to the device
        t = threading.Thread(target=work, args=(i,))
        t.start()
        t.join()
    for o in outs:
        assert (o - want).abs().max() <= 2 ** -10 * want.abs().max()
    assert b.gemm_workspace(dev).data_ptr() == b.gemm_workspace(torch.device("cuda")).data_ptr()
    small, big = b.attention_workspace(dev, 1, 4, 128), b.attention_workspace(dev, 300, 64, 128)
    assert big.numel() > small.numel() or big.data_ptr() == small.data_ptr()
    assert b.attention_workspace(dev, 1, 4, 128).data_ptr() == big.data_ptr()
    q, k = torch.randn(2, 4, 128, device=dev).half(), torch.randn(2, 2, 128, device=dev).half()
    pool = torch.zeros(4, 2 * 64 * 64 + 2 * 64 * 4, dtype=torch.uint8, device=dev)
    table = (pool.data_ptr() + torch.arange(4, device=dev) * pool.shape[1]).view(2, 2, 1).contiguous()
    lens = torch.ones(2, dtype=torch.int32, device=dev)
    ref = b.single_query_attention(q, k, k, table, lens, None, 8192, 64, 128, 1, 128, 1e4, True, True, True)
    got = b.single_query_attention(q, k, k, table, lens, None, 8192.0, torch.tensor(64), 128, torch.tensor(1, device=dev), 128, 10000, 1, 1, 1)
    assert torch.equal(ref, got) and (ref - k.repeat_interleave(2, 1)).abs().max() <= 2e-3 * k.abs().max()
