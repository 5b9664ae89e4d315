"""Float32 products whose K is cut into four stretches (2,048 and more): every kernel adds them in the same
order, so a row has the same bits in all of them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 64, 200, 896, 5000])
@pytest.mark.parametrize("k", [2044, 2048, 2052, 2180, 4864, 8448])
def test_rows_have_the_same_bits_in_every_kernel(n, k):
    """1 to 16 rows (a warp per 8 columns), more (32 x 64, 64 x 64 and 128 x 128 tiles, a cluster of CTAs a
    tile from K = 2,048 on) and rows off 16 bytes (the general kernel); bias, accumulation, ragged edges."""
    from minfer_b200.kernels import api as K
    g = torch.Generator(device="cuda").manual_seed(n + k)
    m = 700
    x = torch.randn(m, k, generator=g, device="cuda")
    w = torch.randn(n, k, generator=g, device="cuda") * k ** -0.5
    bias, old = torch.randn(n, generator=g, device="cuda"), torch.randn(m, n, generator=g, device="cuda")
    want = x.double() @ w.double().t() + bias.double()

    def product(rows, accumulate):
        out = old[rows].clone()
        K.gemm_simt(x[rows].contiguous(), w, bias, out, accumulate)
        return out

    whole = {a: product(slice(0, m), a) for a in (False, True)}
    # 32-bit sums of k products: 2^-24 a step, in four chains of at most k / 4 + 128
    assert float((whole[False].double() - want).abs().max()) < 2 ** -24 * (k / 4 + 131) * float(want.abs().max())
    for rows in (slice(0, 1), slice(3, 7), slice(5, 13), slice(100, 116), slice(1, 41), slice(200, 400)):
        for a in (False, True):
            assert torch.equal(product(rows, a), whole[a][rows]), (rows, a)
    # rows that do not start on 16 bytes
    odd_x, odd_w = torch.zeros(40, k + 1, device="cuda"), torch.zeros(n, k + 1, device="cuda")
    odd_x[:, :k], odd_w[:, :k] = x[:40], w
    out = torch.empty(40, n, device="cuda")
    K.gemm_simt(odd_x[:, :k], odd_w[:, :k], bias, out, False)
    assert torch.equal(out, whole[False][:40])


@pytest.mark.parametrize("k", [40, 2044, 2047, 2048, 2049, 2180, 4864])
@pytest.mark.parametrize("m,n", [(3, 70), (100, 129)])
def test_mixed_types_have_the_bits_of_float32(m, n, k):
    """The general kernel, one stretch of k and four, its last round of two tiles of k whole or half: numbers that
    both types hold give the sums of the float32 kernels."""
    from minfer_b200.kernels import api as K
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    w = (torch.randn(n, k, generator=g, device="cuda") * k ** -0.5).bfloat16()
    old = torch.randn(m, n, generator=g, device="cuda")
    for accumulate in (False, True):
        want = old.clone()
        K.gemm_simt(x.float(), w.float(), None, want, accumulate)
        for a, b in ((x, w), (x, w.float()), (x.float(), w)):
            out = old.clone()
            K.gemm_simt(a, b, None, out, accumulate)
            assert torch.equal(out, want)
    half = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    K.gemm_simt(x, w.float(), None, half, False)
    K.gemm_simt(x.float(), w.float(), None, want, False)
    assert torch.equal(half, want.bfloat16())


@pytest.mark.parametrize("m,n,k,cut", [(485, 2173, 2180, (0, 1)), (390, 9001, 2052, (0, 2)), (700, 900, 2052, (1, 1)),
                                       (1600, 1157, 2052, (1, 2)), (64, 899, 2052, (2, 1)), (41, 12001, 2052, (2, 2))])
def test_every_tile_in_both_forms(m, n, k, cut):
    """Rows, columns and the last stretch end inside a tile: bias and accumulation, the bits of up to 16 rows,
    a guard around the output."""
    from minfer_b200.kernels import api as K
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert K.gemm_f32_cut(m, n, k, 148) == cut
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g, device="cuda")
    w = torch.randn(n, k, generator=g, device="cuda") * k ** -0.5
    bias, old = torch.randn(n, generator=g, device="cuda"), torch.randn(m, n, generator=g, device="cuda")
    want = x.double() @ w.double().t() + bias.double()
    for accumulate in (False, True):
        room = torch.full((m + 2, n + 3), 5.0, device="cuda")
        out = room[1:m + 1, :n]
        out.copy_(old)
        K.gemm_simt(x, w, bias, out, accumulate)
        whole = want + old.double() if accumulate else want
        # as above, and one rounding of the largest value for each addition behind the products
        assert float((out.double() - whole).abs().max()) < 2 ** -24 * (k / 4 + 133) * float(whole.abs().max())
        assert float((room[0] - 5).abs().max()) == float((room[m + 1] - 5).abs().max()) == 0.0
        assert float((room[:, n:] - 5).abs().max()) == 0.0
        for lo in (0, m // 2, m - 9):
            few = old[lo:lo + 9].clone()
            K.gemm_simt(x[lo:lo + 9], w, bias, few, accumulate)
            assert torch.equal(few, out[lo:lo + 9])


@pytest.mark.parametrize("m,n,k", [(5, 896, 4864), (64, 896, 4864), (41, 12001, 2052), (390, 9001, 2052)])
def test_products_of_a_long_k_wait_for_the_kernel_that_writes_their_input(m, n, k):
    """Launched while a norm still writes the rows it reads: up to 16 rows, a cluster a tile, four stretches a CTA."""
    from minfer_b200.kernels import api as K
    g = torch.Generator(device="cuda").manual_seed(m)
    h, w = torch.randn(m, k, generator=g, device="cuda"), torch.randn(n, k, generator=g, device="cuda")
    scale = torch.rand(k, generator=g, device="cuda")
    x, out = torch.empty(m, k, device="cuda"), torch.empty(m, n, device="cuda")
    K.rmsnorm(h, scale, 1e-5, x)
    torch.cuda.synchronize()
    K.gemm_simt(x, w, None, out)
    torch.cuda.synchronize()
    want = out.clone()
    for _ in range(20):
        x.fill_(float("nan"))
        K.rmsnorm(h, scale, 1e-5, x)
        K.gemm_simt(x, w, None, out)
        assert torch.equal(out, want)
