"""The CPython binding behind the operators: what is refused before anything is launched (CPU), and on the GPU that a call lands on the current stream of
its tensors' device, takes whatever int() and float() take, raises what torch's own functions raise, and shares the work spaces that the Python functions
hand out."""
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


def _attention_arguments(device="cpu"):
    """The 16 arguments of single_query_attention_quant; checks of its tensors' shapes and numbers come ahead of the check of the device."""
    q, k = torch.zeros(1, 4, 128, dtype=HALF, device=device), torch.zeros(1, 2, 128, dtype=HALF, device=device)
    lens, s = torch.ones(1, dtype=torch.int32, device=device), torch.zeros(1, dtype=HALF, device=device)
    return [q, k, k, torch.zeros(1, 2, 1, dtype=torch.int64, device=device), lens, 8192, 64, 128, 1, 128, 1e4, True, True,
            torch.zeros(1, 512, dtype=torch.int8, device=device), s, None]


@pytest.mark.parametrize("at,value,error", [
    (3, torch.tensor(0), IndexError),                              # too few dimensions: as tensor.size() and tensor.stride() raise it
    (0, torch.zeros(4, 128, dtype=HALF), IndexError),
    (1, torch.zeros(256, dtype=HALF), IndexError),
    (10, "1e4", RuntimeError), (10, torch.tensor(1e4), RuntimeError), (10, 10000, RuntimeError),  # whatever float() takes: only the device is refused
    (10, "ten", ValueError), (10, None, TypeError),
    (5, "8192", RuntimeError), (5, 8192.7, RuntimeError), (5, 1 << 70, RuntimeError), (5, "x", ValueError), (5, None, TypeError),
])
def test_conversions_and_error_classes(at, value, error):
    from qserve_b200 import backend as b

    args = _attention_arguments()
    args[at] = value
    with pytest.raises(error) as e:
        b.single_query_attention_quant(*args)
    assert e.type is error and (error is not RuntimeError or str(e.value) == "q must be on CUDA")


@pytest.mark.gpu
def test_refusals_on_the_device(dev):
    from qserve_b200 import backend as b

    x, w, o = (torch.zeros(2, 128, dtype=torch.int8, device=dev), torch.zeros(128, 64, dtype=torch.int8, device=dev), torch.zeros(2, 128, dtype=HALF, device=dev))
    s, half = torch.ones(128, dtype=HALF, device=dev), torch.zeros(2, 128, dtype=HALF, device=dev)
    with pytest.raises(IndexError):
        b.w4a8_per_chn_gemm_forward_cuda(x[0], w, s, s, s, s, o)
    with pytest.raises(RuntimeError, match="kernel shape \\(3\\) does not match"):
        b.w8a8_gemm_forward_cuda(x, torch.zeros(3, dtype=torch.int8, device=dev), s, s, o)
    for i in (2, 3, 4, 5):  # a scale, a sum or a zero point that is missing
        args = [x, w, s, s, s, s, o]
        args[i] = None
        with pytest.raises(TypeError):
            b.w4a8_per_chn_gemm_forward_cuda(*args)
    codes, scale = torch.full((2, 128), 7, dtype=torch.int8, device=dev), torch.zeros(2, dtype=HALF, device=dev)
    with pytest.raises(RuntimeError, match="null tensor"):  # no room for the sums: not taken for the form without them
        b.invoke_quant_fuse_sum(codes, half, torch.empty(0, dtype=HALF, device=dev), scale)
    assert (codes == 7).all()
    before = b.attention_workspace(dev, 1, 4, 128)
    with pytest.raises(torch.OutOfMemoryError):  # 10^12 bytes
        b.attention_workspace(dev, 1 << 20, 64, 128)
    assert b.attention_workspace(dev, 1, 4, 128).data_ptr() == before.data_ptr()


@pytest.mark.gpu
def test_a_call_lands_on_the_current_stream(dev):
    """Under capture on a side stream a call writes nothing until the graph is replayed; a launch on any other stream would write at once or break the
    capture."""
    from qserve_b200 import backend as b

    g = torch.Generator(device=dev).manual_seed(1)
    x = torch.randn(3, 256, device=dev, generator=g).half()
    out, eager = torch.zeros(3, 128, dtype=HALF, device=dev), torch.zeros(3, 128, dtype=HALF, device=dev)
    b.silu_and_mul(eager, x)
    graph, st = torch.cuda.CUDAGraph(), torch.cuda.Stream(dev)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=st):
        b.silu_and_mul(out, x)
    torch.cuda.synchronize()
    assert (out == 0).all()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, eager) and (eager != 0).any()
    # and in order with the work queued there: the input is written behind a long chain of products on the side stream
    out.zero_()
    late, m = torch.zeros_like(x), torch.randn(4096, 4096, device=dev)
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        for _ in range(10):
            m = m @ m * 1e-3
        late.copy_(x)
        b.silu_and_mul(out, late)
    st.synchronize()
    assert torch.equal(out, eager)


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
    from qserve_b200._lib import lib

    small = b.attention_workspace(dev, 1, 4, 128)
    assert small.numel() >= lib.qs_attention_workspace_bytes(1, 4, 128)
    per_sequence = lib.qs_attention_workspace_bytes(2, 64, 128) - lib.qs_attention_workspace_bytes(1, 64, 128)
    batch = small.numel() // per_sequence + 2  # more than it has had to hold so far
    old, size = small.data_ptr(), small.numel()
    big = b.attention_workspace(dev, batch, 64, 128)
    assert big.numel() >= lib.qs_attention_workspace_bytes(batch, 64, 128) > size
    assert b.attention_workspace(dev, 1, 4, 128).data_ptr() == big.data_ptr()
    del small  # the outgrown one stays: a graph may hold its address
    for n in (size, size // 2, 512):
        t = torch.empty(n, dtype=torch.uint8, device=dev)
        assert t.data_ptr() + n <= old or t.data_ptr() >= old + size
    q, k = torch.randn(2, 4, 128, device=dev).half(), torch.randn(2, 2, 128, device=dev).half()
    pool = torch.zeros(4, 2 * 64 * 64 + 2 * 64 * 4, dtype=torch.uint8, device=dev)
    table = (pool.data_ptr() + torch.arange(4, device=dev) * pool.shape[1]).view(2, 2, 1).contiguous()
    lens = torch.ones(2, dtype=torch.int32, device=dev)
    ref = b.single_query_attention(q, k, k, table, lens, None, 8192, 64, 128, 1, 128, 1e4, True, True, True)
    got = b.single_query_attention(q, k, k, table, lens, None, 8192.0, torch.tensor(64), 128, torch.tensor(1, device=dev), 128, 10000, 1, 1, 1)
    assert torch.equal(ref, got) and (ref - k.repeat_interleave(2, 1)).abs().max() <= 2e-3 * k.abs().max()
