"""Row operations over prompts: the kernels that take many rows at once give every row the bits that the kernels for few rows give it (norm and quantisation,
with and without the fused sum), at their edges: the smallest number of rows that takes them, rows of one vector, of a part of the lanes, of every lane,
widths around the reference's 1024 threads.  Rotary + append: a packed buffer that does not start on an 8-byte boundary, more head rows than one batch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [8, 248, 256, 264, 1000, 1024, 1032, 2048, 4088, 4096])
@pytest.mark.parametrize("rows", [592, 1185])
def test_many_rows_have_the_bits_of_few(dev, rows, H):
    import qserve_backend.fused_kernels as fk
    import qserve_backend.layernorm_ops as ln

    g = torch.Generator(device=dev).manual_seed(rows + H)
    x = (torch.randn(rows, H, device=dev, generator=g) * 3).half()
    x[0] = 0
    gamma = torch.randn(H, device=dev, generator=g).half()

    def run(piece):
        out = []
        for op in range(4):
            q, s, t = torch.zeros(rows, H, dtype=torch.int8, device=dev), torch.zeros(rows, dtype=torch.half, device=dev), torch.zeros(rows, dtype=torch.half, device=dev)
            for a in range(0, rows, piece):
                r = slice(a, a + piece)
                if op == 0:
                    ln.rms_norm_general(q[r], x[r], gamma, s[r], 1e-5, True)
                elif op == 1:
                    ln.rms_norm_general_fuse_sum(q[r], x[r], gamma, t[r], s[r], 1e-5, True)
                elif op == 2:
                    fk.invoke_quant(q[r], x[r], s[r])
                else:
                    fk.invoke_quant_fuse_sum(q[r], x[r], t[r], s[r])
            out += [q, s, t]
        return out

    for a, b in zip(run(rows), run(200)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("H", [8, 1032, 4096])
@pytest.mark.parametrize("rows", [1399, 1400])
def test_many_rows_with_the_sum(dev, rows, H):
    test_many_rows_have_the_bits_of_few(dev, rows, H)  # quantisation with the sum: a warp per row from 1400 rows on


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("Hq,Hkv", [(1, 1), (3, 3), (32, 8), (40, 8), (32, 32)])
def test_append_of_an_unaligned_buffer(dev, bits, Hq, Hkv):
    import qserve_backend.fused_attention as fa

    D, lens = 128, [70, 1, 130]
    T, width, blocks = sum(lens), (Hq + 2 * Hkv) * 128, 3
    g = torch.Generator(device=dev).manual_seed(Hq + bits)
    base = torch.randn(T * width + 2, device=dev, generator=g).half()
    code = Hkv * 64 * D * bits // 8
    lens_d = torch.tensor(lens, dtype=torch.int32, device=dev)
    cu = torch.tensor([0, 70, 71, 201], dtype=torch.int32, device=dev)
    got = []
    for shift in (0, 2):  # halves: 0 or 4 bytes past an 8-byte boundary
        qkv = torch.empty(T * width + 2, dtype=torch.half, device=dev)[shift:shift + T * width].view(T, width).copy_(base[:T * width].view(T, width))
        pools = [torch.zeros(len(lens) * blocks, code + Hkv * 64 * 4, dtype=torch.uint8, device=dev) for _ in range(2)]
        at = torch.arange(len(lens) * blocks, device=dev).view(len(lens), blocks)
        table = torch.stack([p.data_ptr() + at * p.shape[1] for p in pools], 1).contiguous()
        pad = fa.compute_padding_offsets(cu, max(lens), T)
        fa.apply_bias_rope_update_kv_cache(qkv, lens_d, pad, table, Hq, Hkv, max(lens), 64, Hkv * D * bits // 8, D, 10000.0, 8192, True, bits == 4, True)
        got.append((qkv, *pools))
    for a, b in zip(*got):
        assert torch.equal(a, b)
    # the rotation in 64 bits: products and sums of fp16 numbers with fp32 sines and cosines (2^-22 of angles up to 130), rounded to fp16
    qkv = base[:T * width].view(T, Hq + 2 * Hkv, D).double()
    pos = torch.cat([torch.arange(n, device=dev) for n in lens]).double()
    angle = pos[:, None, None] * 10000.0 ** (-torch.arange(0, D, 2, device=dev).double() / D)
    lo, hi = qkv[..., :64], qkv[..., 64:]
    want = torch.cat([lo * angle.cos() - hi * angle.sin(), hi * angle.cos() + lo * angle.sin()], -1)
    want[:, Hq + Hkv:] = qkv[:, Hq + Hkv:]
    err = (got[0][0].view(T, -1, D).double() - want).abs()
    assert bool((err <= want.abs() * 2.0 ** -11 + 130 * 2.0 ** -22 * 8).all())
