"""Kernels of a decode step: products of a handful of tokens (``gemm_few_kernel``) and single queries whose
old keys are read before the kernel before them ends."""
import pytest
import torch

from test_furitar_kernels_gpu import _i32, _paged, _qkv_case

pytestmark = pytest.mark.gpu

# the sums are float32 sums of exact bfloat16 products: 2^-24 a step over at most 20,000 of them in several
# chains, relative to the largest value; bfloat16 outputs round once (2^-9)
TOL = {torch.float32: 2e-5, torch.bfloat16: 1e-2}


def _close(got, want):
    err = float((got.double() - want.double()).abs().max() / want.double().abs().max().clamp_min(1e-30))
    assert err < TOL[got.dtype], err


@pytest.fixture
def any_size():
    """The kernel for a handful of tokens takes small products too."""
    from minfer_b200.kernels import api as K
    K.gemm_few_mode(2)
    yield
    K.gemm_few_mode(1)


def _operands(m, n, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    w = (torch.randn(n, k, generator=g, device="cuda") * k ** -0.5).bfloat16()
    return x, w, torch.randn(n, generator=g, device="cuda"), torch.randn(m, n, generator=g, device="cuda")


# (rows of W, k): the CTAs that cut K between them at 1, 3, 8, 9 and 16 tokens; 0: too large beyond 8 tokens, or the
# tokens do not fit shared memory
SIZES = {(8, 8): (1, 1, 1, 1, 1), (14, 72): (1, 1, 1, 1, 1), (250, 328): (1, 1, 1, 1, 1), (1152, 896): (1, 1, 1, 1, 1),
         (896, 4864): (1, 1, 1, 1, 2), (2048, 8448): (1, 1, 1, 0, 0), (9728, 896): (1, 1, 1, 0, 0),
         (1001, 13824): (1, 1, 2, 0, 0), (40, 20000): (4, 4, 4, 4, 0),
         # several row tiles a CTA for two tiles of tokens as well; many, of a k that one warp or two have
         (2500, 1032): (1, 1, 1, 1, 1), (5000, 328): (1, 1, 1, 1, 1), (9001, 264): (1, 1, 1, 1, 1),
         (17472, 128): (1, 1, 1, 1, 1), (88, 4496): (2, 2, 2, 2, 2)}


@pytest.mark.parametrize("m", [1, 3, 8, 9, 16])
@pytest.mark.parametrize("n,k", list(SIZES))
def test_products_of_a_handful_of_tokens(m, n, k, any_size):
    """Row tiles that end inside a tile, K that ends inside a unit, K cut between the CTAs of a cluster, a
    warp or a CTA without k; every epilogue, the norm folded in on both sides; the same bits twice."""
    from minfer_b200.kernels import api as K
    parts = K.gemm_few_groups(m, n, k)
    cluster = SIZES[n, k][(1, 3, 8, 9, 16).index(m)]
    assert K.gemm_few_plan(m, n, k, 148)[1] == cluster
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert (parts > 0) == (cluster > 0)
    if parts == 0:
        pytest.skip("left to other kernels")
    x, w, bias, h0 = _operands(m, n, k, m + n + k)
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    want = x.double() @ w.double().t()
    out = torch.full((m, n), float("nan"), device="cuda")
    K.gemm_tc(x, w, bias, out, K.EPI_STORE, st)
    _close(out, want + bias.double())
    again = torch.empty_like(out)
    K.gemm_tc(x, w, bias, again, K.EPI_STORE, st)
    assert torch.equal(out, again)
    half = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    K.gemm_tc(x, w, None, half, K.EPI_STORE, st)
    _close(half, want)
    # the residual completed and the next norm prepared, a guard behind what is written
    gw = 1 + 0.1 * bias
    h, ssq = h0.clone(), torch.full((parts + 1, m), float("nan"), device="cuda")
    xp = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    K.gemm_tc_fused(x, w, bias, h, K.EPI_ACCUM, st, prep_x=xp, prep_weight=gw, prep_ssq=ssq[:parts])
    _close(h, h0.double() + want + bias.double())
    _close(xp, h.double() * gw.double())
    assert torch.isnan(ssq[parts]).all()
    _close(ssq[:parts].sum(0), (h.double() ** 2).sum(-1))
    added = h0.clone()
    K.gemm_tc(x, w, None, added, K.EPI_ACCUM, st)
    _close(added, h0.double() + want)
    # a row scale, the gated and the dense activations
    sums = torch.rand(5, m, device="cuda") * k
    scale = 1.0 / torch.sqrt(sums.double().sum(0) / k + 1e-6)
    y = want * scale[:, None]
    z = torch.empty(m, n, device="cuda")
    K.gemm_tc_fused(x, w, None, z, K.EPI_STORE, st, row_scale=K.RowScale(sums, k, 1e-6))
    _close(z, y)
    K.gemm_tc_xielu(x, w, half, 0.7, 0.9, st, row_scale=K.RowScale(sums, k, 1e-6))
    _close(half, torch.where(y > 0, 0.7 * y * y + 0.5 * y, 0.9 * (torch.expm1(y) - y) + 0.5 * y))
    K.gemm_tc_xielu(x, w, half, 1.0, 0.0, st, act_l=0.0)
    _close(half, torch.relu(want) ** 2)
    if n % 2 == 0:
        act = torch.empty(m, n // 2, dtype=torch.bfloat16, device="cuda")
        for name, p0, p1 in (("silu", 0.0, 0.0), ("gelu_tanh", 0.0, 0.0), ("clamped_swish", 1.5, 1.7)):
            K.gemm_tc_gated(x, w, act, name, p0, p1, st)
            g, u = want[:, 0::2], want[:, 1::2]
            if name == "silu":
                ref = torch.nn.functional.silu(g) * u
            elif name == "gelu_tanh":
                ref = torch.nn.functional.gelu(g, approximate="tanh") * u
            else:
                g, u = g.clamp(max=p0), u.clamp(-p0, p0)
                ref = g * torch.sigmoid(p1 * g) * (u + 1)
            _close(act, ref)
    assert int(st) == 0


def test_products_of_a_handful_of_tokens_take_strided_rows(any_size):
    """Rows of x, W and the outputs further apart than they are long, and an infinite weight."""
    from minfer_b200.kernels import api as K
    m, n, k = 5, 300, 264
    x, w, _, _ = _operands(m, n, k, 3)
    wide_x = torch.zeros(m, k + 40, dtype=x.dtype, device="cuda")
    wide_w = torch.zeros(n, k + 8, dtype=x.dtype, device="cuda")
    wide_x[:, :k], wide_w[:, :k] = x, w
    wide_w[:, k:] = float("inf")              # what lies between two rows is not read
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = torch.zeros(m, n + 3, device="cuda")
    K.gemm_tc(wide_x[:, :k], wide_w[:, :k], None, out[:, :n], K.EPI_STORE, st)
    _close(out[:, :n], x.double() @ w.double().t())
    assert float(out[:, n:].abs().sum()) == 0.0
    wide_w[7, 3] = float("inf")
    K.gemm_tc(wide_x[:, :k], wide_w[:, :k], None, out[:, :n], K.EPI_STORE, st)
    assert not torch.isfinite(out[:, 7]).any() and torch.isfinite(out[:, 8:n]).all() and torch.isfinite(out[:, :7]).all()


@pytest.mark.parametrize("chunk,ring", [(0, 0), (200, 0), (200, 256), (128, 192)])
def test_old_keys_read_early_are_the_same_keys(chunk, ring):
    """One query a sequence at its last position: with and without the promise that older keys are final."""
    from minfer_b200.kernels import api as K
    heads, kv, hd, vd, lengths = 8, 2, 128, 128, [1, 31, 32, 33, 64, 65, 190, 193, 401, 1000]
    q, k, v, r1, r2 = _qkv_case(5, heads, kv, hd, vd, lengths)
    t = torch.bfloat16
    kc, vc, table, stride = _paged(k.to(t), v.to(t), lengths, ring, seed=2)
    kc, vc = kc.cuda(), vc.cuda()
    ends = torch.tensor(lengths).cumsum(0) - 1
    qd = q.to(t)[ends].contiguous().cuda()
    outs = []
    for final in (False, True):
        out = torch.empty(len(lengths), heads * vd, dtype=t, device="cuda")
        K.sink_attention_decode(qd, kc, vc, _i32(list(range(len(lengths)))), _i32([n - 1 for n in lengths]),
                                table.reshape(-1).cuda(), stride, ring, out, r1.float().cuda(), r2.float().cuda(),
                                heads, kv, hd, vd, 0, chunk, True, 0.3, chunk if chunk else max(lengths),
                                old_keys_final=final)
        outs.append(out)
    assert torch.isfinite(outs[0]).all() and torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("width", [4, 200, 2048, 4096, 4100, 30])
@pytest.mark.parametrize("splits", [0, 1, 8, 16, 17])
def test_norm_and_shift_of_one_token_a_row(width, splits):
    """Widths inside and beyond the single-pass form, K splits up to and beyond those it adds, a row at
    position 0, rows that share a state tensor, two steps one behind the other."""
    from minfer_b200.kernels import api as K
    g = torch.Generator(device="cuda").manual_seed(width + splits)
    rows, eps = 5, 1e-5
    slots, positions = _i32([6, 0, 3, 2, 5]), _i32([0, 4, 9, 100, 1])
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")            # noqa: E731
    w, shift, state, bias = 1 + 0.1 * rand(width), rand(width), rand(7, width), rand(width)
    ref_state = state.double().clone()
    for step in range(2):
        x = rand(rows, width)
        part = rand(splits, rows, width) if splits else None
        full = x.double() + (part.double().sum(0) + bias.double() if splits else 0.0)
        pos = positions + step
        y = torch.empty(rows, width, device="cuda")
        K.norm_shift(x, w, shift, eps, pos, _i32(list(range(rows))), _i32(list(range(rows + 1))), slots, state, y,
                     False, partial=part, bias=bias if splits else None)
        n = full / torch.sqrt((full ** 2).mean(-1, keepdim=True) + eps) * w.double()
        before = torch.where(pos[:, None] > 0, ref_state[slots.long()], torch.zeros_like(n))
        _close(y, n + (before - n) * shift.double())
        ref_state[slots.long()] = n
        _close(state, ref_state)
        _close(x, full)


@pytest.mark.parametrize("m,n,k", [(1, 1152, 896), (8, 3072, 2048), (16, 896, 4864), (3, 40, 20000)])
def test_products_of_a_handful_of_tokens_wait_for_the_kernel_that_writes_their_tokens(m, n, k):
    """Launched while a norm still writes the rows it reads: one CTA a row tile, clusters of two and of four."""
    from minfer_b200.kernels import api as K
    assert K.gemm_few_groups(m, n, k) > 0
    g = torch.Generator(device="cuda").manual_seed(m + n)
    h, scale = torch.randn(m, k, generator=g, device="cuda"), torch.rand(k, generator=g, device="cuda")
    w = (torch.randn(n, k, generator=g, device="cuda") * k ** -0.5).bfloat16()
    st = torch.zeros(1, dtype=torch.int32, device="cuda")
    x, out = torch.empty(m, k, dtype=torch.bfloat16, device="cuda"), torch.empty(m, n, device="cuda")
    K.rmsnorm(h, scale, 1e-5, x)
    torch.cuda.synchronize()
    K.gemm_tc(x, w, None, out, K.EPI_STORE, st)
    torch.cuda.synchronize()
    want = out.clone()
    for _ in range(20):
        x.fill_(float("nan"))
        K.rmsnorm(h, scale, 1e-5, x)
        K.gemm_tc(x, w, None, out, K.EPI_STORE, st)
        assert torch.equal(out, want)
    assert int(st) == 0
