"""The products of a few rows (gemm_few.cu) at the edges of their tiles, boxes and rows, against float64 sums of the same bfloat16 operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from llm_b200.csrc import ops
    return ops


def operands(M, N, K, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed + M * 7 + N * 3 + K)
    a = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    return a, w


# K: one block, a box and a ragged one, several steps with a ragged last; N: fewer than SMs, no multiple of a tile, several tiles a CTA
SIZES = [(96, 64), (17, 512), (2369, 576), (300, 1408), (2560, 2048), (5000, 2624)]
# more passes of the loops that stage the rows (64 blocks of 64 a pass), the second one ragged, whole, and up to four; few outputs, to keep it quick
LONG = [(1, 300, 4160), (3, 300, 4160), (1, 100, 5632), (8, 100, 5632), (1, 64, 14336), (3, 64, 14336)]


def bound(K):
    """Of the distance from the exact sum, as a share of the sum of the terms' absolute values: an accumulator takes 2 MMAs of each of its warp's blocks, a
    block of 64 k in every 512, and each may cut off 2^-23 of what it has; two accumulators, eight warps and the factor behind them: ten roundings."""
    return (2 * -(-K // 512) + 10) * 2.0 ** -23


@pytest.mark.parametrize("M,N,K", [(m, n, k) for m in (1, 3, 7, 8) for n, k in SIZES] + LONG)
def test_sums(ops, M, N, K):
    a, w = operands(M, N, K)
    assert ops.gemm_few_available(a, w, M)
    exact = a.double() @ w.double().T
    scale = (a.double().abs() @ w.double().abs().T)
    out = torch.full((M + 1, N + 3), 7.0, device=DEV)
    ops.gemm_few(a, w, out[:, :N], M)
    assert bool(((out[:M, :N].double() - exact).abs() <= bound(K) * scale + 1e-30).all())
    assert bool((out[M] == 7).all()) and bool((out[:, N:] == 7).all())            # nothing beside the results
    half = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    ops.gemm_few(a, w, half, M)
    assert torch.equal(half, out[:M, :N].to(torch.bfloat16))
    resid = torch.randn(M, N, device=DEV)
    added = resid.clone()
    ops.gemm_few(a, w, added, M, kind="add")
    assert torch.equal(added, resid + out[:M, :N])


@pytest.mark.parametrize("M", [1, 5, 8])
@pytest.mark.parametrize("N,K", [(34, 64), (2370, 576), (1408, 2048)])
@pytest.mark.parametrize("act", ["silu", "relu"])
def test_gated(ops, M, N, K, act):
    a, w = operands(M, 2 * N, K)
    z = a.double() @ w.double().T
    scale = a.double().abs() @ w.double().abs().T
    g, u = z[:, :N], z[:, N:]
    ref = (torch.nn.functional.silu(g) if act == "silu" else torch.relu(g)) * u
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    ops.gemm_few(a, w, out, M, kind=act)
    # one rounding of the result, and the sums' errors through a product whose factors have slopes of at most 1.1
    slack = 2.0 ** -8 * ref.abs() + 1.2 * bound(K) * (scale[:, :N] * u.abs() + scale[:, N:] * g.abs()) + 1e-12
    assert bool(((out.double() - ref).abs() <= slack).all())


# under a norm a pass takes 32 blocks: K of one pass, of a second one of one block, of two whole ones, of a third; the last: a stage of a single box beside
# the rows, tiles of 16
NORMED = [(m, n, k) for m in (1, 2, 8) for n, k in ((40, 64), (300, 1408), (2560, 2048), (200, 2112), (96, 4096), (40, 4160))] + [(8, 2368, 7168)]


@pytest.mark.parametrize("M,N,K", NORMED)
def test_rows_under_a_norm(ops, M, N, K):
    _, w = operands(M, N, K)
    x = torch.randn(M + 2, K, device=DEV) * torch.tensor([0.01, 300.0] * (M + 2), device=DEV)[:M + 2, None]
    gain = 1.0 + 0.1 * torch.randn(K, device=DEV)
    out = torch.empty(M, N, device=DEV)
    ops.gemm_few(ops.NormedRows(x, gain, 1e-5, M, torch.bfloat16), w, out, M)
    xd = x[:M].double()
    h = xd / torch.sqrt((xd * xd).mean(-1, keepdim=True) + 1e-5) * gain.double()
    # one rounding to bfloat16 (2^-9 of each) of what multiplies the weights, the rest in float32
    scale = h.abs() @ w.double().abs().T
    assert bool(((out.double() - h @ w.double().T).abs() <= (2.0 ** -9 + 1e-5) * scale).all())


@pytest.mark.parametrize("M", [1, 5, 8])
@pytest.mark.parametrize("N,K", [(34, 64), (300, 2048), (200, 2112), (1190, 4096), (40, 4160)])
@pytest.mark.parametrize("act", ["silu", "relu", "clamped"])
def test_gated_on_rows_under_a_norm(ops, M, N, K, act):
    """The form of a decode step's feed-forward: the norm before the product and the activation behind it."""
    _, w = operands(M, 2 * N, K)
    x = torch.randn(M, K, device=DEV) * torch.tensor([0.01, 300.0, 1.0] * M, device=DEV)[:M, None]
    gain = 1.0 + 0.1 * torch.randn(K, device=DEV)
    bias = torch.randn(2 * N, device=DEV) if act == "clamped" else None
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    ops.gemm_few(ops.NormedRows(x, gain, 1e-5, M, torch.bfloat16), w, out, M, kind=act, bias=bias, limit=1.5, alpha=1.702)
    xd = x.double()
    h = xd / torch.sqrt((xd * xd).mean(-1, keepdim=True) + 1e-5) * gain.double()
    z = h @ w.double().T + (bias.double() if bias is not None else 0)
    err = (2.0 ** -9 + 1e-5) * (h.abs() @ w.double().abs().T)           # of the two sums: what multiplies the weights is rounded once to bfloat16
    (g, u), (eg, eu) = z.chunk(2, -1), err.chunk(2, -1)
    if act == "clamped":
        g, u = g.clamp(max=1.5), u.clamp(-1.5, 1.5) + 1
        f = g * torch.sigmoid(1.702 * g)
    else:
        f = torch.nn.functional.silu(g) if act == "silu" else torch.relu(g)
    # the activations have slopes of at most 1.2 and |f| <= |g| (clamped: 1.2 |g|)
    slack = 2.0 ** -8 * (f * u).abs() + 1.2 * (eg * u.abs() + eu * g.abs() + eg * eu) + 1e-6
    assert bool(((out.double() - f * u).abs() <= slack).all())


@pytest.mark.parametrize("M", [1, 8])
@pytest.mark.parametrize("N,K", [(34, 64), (2370, 576), (1408, 2048)])
@pytest.mark.parametrize("biased", [False, True])
def test_clamped_unit_and_biases(ops, M, N, K, biased):
    a, w = operands(M, 2 * N, K)
    bias = torch.randn(2 * N, device=DEV) if biased else None
    z = a.double() @ w.double().T + (bias.double() if biased else 0)
    scale = a.double().abs() @ w.double().abs().T
    limit, alpha = 1.5, 1.702
    g, u = z[:, :N].clamp(max=limit), z[:, N:].clamp(-limit, limit)
    ref = g * torch.sigmoid(alpha * g) * (u + 1)
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    ops.gemm_few(a, w, out, M, kind="clamped", bias=bias, limit=limit, alpha=alpha)
    # slopes: the gate's function of at most 1.1 in the range that is clamped above, the linear branch's factor of at most 2.5
    slack = 2.0 ** -8 * ref.abs() + 3 * bound(K) * (scale[:, :N] + scale[:, N:] * g.abs()) + 1e-6
    assert bool(((out.double() - ref).abs() <= slack).all())
    rows = torch.empty(M, 2 * N, device=DEV)
    ops.gemm_few(a, w, rows, M, bias=bias)
    assert bool(((rows.double() - z).abs() <= bound(K) * (scale + 1)).all())


def test_what_is_not_taken(ops):
    a, w = operands(8, 64, 128)
    assert not ops.gemm_few_available(a.float(), w.float(), 8)
    assert not ops.gemm_few_available(torch.cat([a, a]), w, 9)                    # more than eight rows
    assert not ops.gemm_few_available(a[:, :96], w[:, :96], 8)                    # K off the 64-grid
    assert not ops.gemm_few_available(a[:, 4:68], w[:, :64], 8)                   # rows off the 16-byte grid
    assert not ops.gemm_few_takes(8, 16384)                                       # rows that leave no room for the stages
    for rows in range(0, 18):
        for k in (64, 96, 2048, 4096, 5632, 14336, 16384, 65536):
            assert bool(ops.load_tensor().llmk_gemm_few_supported(rows, k)) == ops.gemm_few_takes(rows, k), (rows, k)


def test_two_threads_with_products_of_different_sizes(ops):
    """Each launch takes the shared memory that its rows and stages need, whatever another thread launches at the same time; a product may be a
    thread's first call into CUDA."""
    import threading
    small, large = operands(1, 96, 64), operands(8, 2368, 5632)
    want = [ops.gemm_few(a, w, torch.empty(a.shape[0], w.shape[0], device=DEV), a.shape[0]) for a, w in (small, large)]
    outs, errors = [torch.empty_like(t) for t in want], []

    def loop(a, w, out):
        try:
            for _ in range(3000):
                ops.gemm_few(a, w, out, a.shape[0])
        except Exception as e:      # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(a, w, o)) for (a, w), o in zip((small, large), outs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors and all(torch.equal(o, t) for o, t in zip(outs, want))


@pytest.mark.parametrize("M,N,K", [(1, 148, 2048), (8, 2368, 5632), (8, 1184, 7168)])
def test_behind_a_kernel_that_takes_longer_than_the_waits(ops, M, N, K):
    """The kernel starts under the one before it and asks for weights; its bounded waits (2e9 cycles, a second) count from that one's end."""
    a, w = operands(M, N, K)
    want = ops.gemm_few(a, w, torch.empty(M, N, device=DEV), M)
    x, y = torch.ones(1, 40_000_001, device=DEV), torch.ones(1, 40_000_001, device=DEV)      # one tile, a long chain of k
    one, out = torch.empty(1, 1, device=DEV), torch.empty(M, N, device=DEV)
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    begin.record()
    ops.gemm_simt(x, y, one, 1)
    ops.gemm_few(a, w, out, M)
    end.record()
    torch.cuda.synchronize()
    assert begin.elapsed_time(end) > 1200
    assert ops.gemm_tc_take_error() == 0 and torch.equal(out, want)
