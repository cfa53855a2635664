"""Products that fit one wave of thread blocks: the weight stream for up to 8 rows (16-bit and 4-bit weights) and the small tiles with
their k range over a cluster, at the edges of their units, steps, tiles and splits."""

import pytest
import torch

from mllm_b200 import ops

pytestmark = pytest.mark.gpu

# the result is rounded to 8 bits (bf16), by at most 2^-9 of itself
TOLERANCE = 2 ** -8


def _rand(*shape, seed=0, std=1.0, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * std).to(dtype)


def _close(got, want):
    error = (got.double() - want).norm() / want.norm()
    assert error < TOLERANCE, float(error)
    assert torch.isfinite(got.float()).all()


# n: part of a unit of 16 rows, several units per block; k: less than the eight warps' steps, a last step that some warps lack,
# registers' limit (4096), two and eight blocks of a cluster
@pytest.mark.parametrize("n,k", [(8, 32), (24, 96), (1000, 544), (4096, 4096), (520, 4128), (264, 12288), (40, 32768), (9472, 512)])
@pytest.mark.parametrize("m", [1, 3, 8])
def test_stream(m, n, k):
    x, w = _rand(m, k), torch.nn.Parameter(_rand(n, k, seed=1, std=0.05), requires_grad=False)
    _close(ops.linear(x, w), x.double() @ w.double().t())
    b, r = _rand(n, seed=2), _rand(m, n, seed=3)
    _close(ops.linear(x, w, b, r), x.double() @ w.double().t() + b.double() + r.double())


# 9 rows and more: every width of a tile, part of a tile in each direction, every split of k, a k that is no multiple of 64
@pytest.mark.parametrize("n,k", [(8, 64), (136, 520), (1024, 2048), (1000, 544), (4096, 4096), (384, 8192)])
@pytest.mark.parametrize("m", [9, 16, 17, 33, 65, 129, 256, 300, 784])
def test_tiles(m, n, k):
    x, w = _rand(m, k), torch.nn.Parameter(_rand(n, k, seed=1, std=0.05), requires_grad=False)
    _close(ops.linear(x, w), x.double() @ w.double().t())
    b, r = _rand(n, seed=2), _rand(m, n, seed=3)
    _close(ops.linear(x, w, b, r), x.double() @ w.double().t() + b.double() + r.double())


@pytest.mark.parametrize("n,k", [(256, 64), (2048, 1024), (512, 4160), (768, 12288)])
@pytest.mark.parametrize("m", [1, 8, 20, 100, 300])
def test_gated(m, n, k):
    x, w = _rand(m, k), torch.nn.Parameter(_rand(n, k, seed=1, std=0.05), requires_grad=False)
    y = (x.double() @ w.double().t()).view(m, -1, 2, ops.SWIGLU_BLOCK)
    _close(ops.linear_swiglu(x, w), (torch.nn.functional.silu(y[:, :, 0]) * y[:, :, 1]).reshape(m, -1))


# the bias is written by a kernel that lets the product start before it has stored anything, while a product in front still reads
# what was there
@pytest.mark.parametrize("m,act", [(4, None), (20, None), (64, None), (200, None), (64, "clamped"), (600, "clamped")])
def test_bias_of_the_kernel_in_front(m, act):
    n = k = 4096
    x, w = _rand(m, k), torch.nn.Parameter(_rand(n, k, seed=1, std=0.01), requires_grad=False)
    gain, src, bias = torch.ones(n, device="cuda", dtype=torch.bfloat16), _rand(1, n, seed=9), _rand(n, seed=10)

    def product(b):
        return ops.linear(x, w, b) if act is None else ops.linear_swiglu(x, w, act=act, bias=b, limit=7.0)

    product(bias)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        product(bias)
        ops.ext().rmsnorm(src, gain, bias.view(1, n), 1e-6)
        got = product(bias)
    for i in range(20):
        src.copy_(_rand(1, n, seed=11 + i))
        want = product(ops.rmsnorm(src, gain, 1e-6).view(n).clone())
        graph.replay()
        assert torch.equal(got, want)


@pytest.mark.parametrize("m", [9, 40, 200, 400])
def test_tiles_int8(m):
    n, k = 328, 1056
    g = torch.Generator(device="cuda").manual_seed(5)
    a, w = (torch.randint(-127, 128, (r, k), generator=g, device="cuda", dtype=torch.int8) for r in (m, n))
    sa, sw = (torch.rand((r,), generator=g, device="cuda") * 0.01 + 0.001 for r in (m, n))
    _close(ops.int8_scaled_mm(a, w, sa, sw, torch.bfloat16), (a.double() @ w.double().t()) * sa.double()[:, None] * sw.double())


@pytest.mark.parametrize("m", [9, 64, 200, 300])
def test_int8_sums_are_whole(m):
    """Parts of a split k that cancel: whole numbers of 27 bits whose sum is small."""
    n, k = 136, 16384
    a = torch.full((m, k), 127, device="cuda", dtype=torch.int8)
    w = torch.full((n, k), 127, device="cuda", dtype=torch.int8)
    w[:, k // 2:] = -127
    w[:, -1] = -126
    g = torch.Generator(device="cuda").manual_seed(5)
    a[:, :k // 2 - 1] -= torch.randint(0, 2, (m, k // 2 - 1), generator=g, device="cuda", dtype=torch.int8)
    a[:, k // 2:-1] = a[:, :k // 2 - 1]
    one_a, one_w = torch.ones(m, device="cuda"), torch.ones(n, device="cuda")
    got = ops.int8_scaled_mm(a, w, one_a, one_w, torch.bfloat16)
    assert torch.equal(got, (a.double() @ w.double().t()).to(torch.bfloat16))


@pytest.mark.parametrize("n,k,group", [(8, 128, 128), (1000, 1280, 128), (4096, 4096, 128), (264, 12288, 256), (40, 2048, 2048), (136, 2048, 64)])
@pytest.mark.parametrize("m", [1, 5, 8])
@pytest.mark.parametrize("zeros,interleaved", [(False, True), (True, True), (True, False), (False, False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_stream_4bit(m, n, k, group, zeros, interleaved, dtype):
    g = torch.Generator(device="cuda").manual_seed(n + k)
    words = torch.randint(-2 ** 31, 2 ** 31, (n, k // 8), generator=g, device="cuda", dtype=torch.int32)
    scale = (torch.rand((n, k // group), generator=g, device="cuda") * 0.01 + 0.005).to(dtype)
    z = torch.randint(0, 16, (n, k // group), generator=g, device="cuda", dtype=torch.uint8) if zeros else None
    x = _rand(m, k, dtype=dtype)
    codes = ((words.unsqueeze(-1) >> torch.arange(0, 32, 4, device="cuda", dtype=torch.int32)) & 15).flatten(1).double().view(n, -1, group)
    w = ((codes - (8 if z is None else z.double().unsqueeze(-1))) * scale.double().unsqueeze(-1)).flatten(1)
    _close(ops.w4a16_gemm(x, ops.w4a16_interleave(words) if interleaved else words, scale, z, group, None, interleaved=interleaved), x.double() @ w.t())


@pytest.mark.parametrize("zeros,interleaved", [(False, True), (True, True), (True, False), (False, False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_stream_4bit_large_values(zeros, interleaved, dtype):
    n, k, group, m = 264, 4096, 128, 5
    g = torch.Generator(device="cuda").manual_seed(n + k)
    words = torch.randint(-2 ** 31, 2 ** 31, (n, k // 8), generator=g, device="cuda", dtype=torch.int32)
    scale = (torch.rand((n, k // group), generator=g, device="cuda") * 0.01 + 0.005).to(dtype)
    z = torch.randint(0, 16, (n, k // group), generator=g, device="cuda", dtype=torch.uint8) if zeros else None
    x = _rand(m, k, dtype=dtype)
    # infinities and NaN are those of the products; sums have the size of the result, so x may be as large as the type allows
    x[1, 77] = float("inf")
    x[2, 900] = -float("inf")
    x[3, 5] = float("nan")
    if dtype == torch.bfloat16:
        x[4] *= 1e37
    codes = ((words.unsqueeze(-1) >> torch.arange(0, 32, 4, device="cuda", dtype=torch.int32)) & 15).flatten(1).double().view(n, -1, group)
    w = ((codes - (8 if z is None else z.double().unsqueeze(-1))) * scale.double().unsqueeze(-1)).flatten(1)
    got = ops.w4a16_gemm(x, ops.w4a16_interleave(words) if interleaved else words, scale, z, group, None, interleaved=interleaved)
    want = x.double() @ w.t()
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[1:3].isinf() & (got[1:3] > 0), want[1:3].isinf() & (want[1:3] > 0))
    _close(got[[0, 4]], want[[0, 4]])
