"""Each kernel alone against a plain float64 torch restatement, at sizes
other than the engine's (widths and vocabularies that are no power of two,
head sizes in steps of 16, odd head counts)."""
import math

import pytest
import torch

from brolm_b200 import kernels
from tests.plain import gemma2_plain as plain

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TOL = {torch.float32: 2e-6, torch.bfloat16: 8e-3}   # relative to the largest magnitude of the result


def close(got, ref, dtype, scale=None):
    ref = ref.double().cpu()
    got = got.double().cpu()
    s = scale if scale is not None else max(1e-30, float(ref.abs().max()))
    err = float((got - ref).abs().max()) / s
    assert err <= TOL[dtype], f"error {err:.3e} exceeds {TOL[dtype]:.1e}"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_embed_scale(dtype):
    g = torch.Generator().manual_seed(0)
    table = torch.randn(1000, 200, generator=g).to(dtype)
    ids = torch.randint(0, 1000, (37,), generator=g, dtype=torch.int32)
    out = torch.empty(37, 200, dtype=torch.float32, device=DEV)
    kernels.embed_scale(ids.to(DEV), table.to(DEV), math.sqrt(200.0), out)
    ref = plain.embed(table, ids, 200)
    close(out, ref, torch.float32)


@pytest.mark.parametrize("xd,wd,od", [(torch.float32, torch.float32, torch.float32),
                                       (torch.float32, torch.bfloat16, torch.bfloat16),
                                       (torch.bfloat16, torch.float32, torch.bfloat16),
                                       (torch.float32, torch.float32, torch.bfloat16)])
@pytest.mark.parametrize("hidden", [200, 2304])
def test_rmsnorm(xd, wd, od, hidden):
    g = torch.Generator().manual_seed(1)
    x = (torch.randn(19, hidden, generator=g) * 3).to(xd)
    w = (torch.randn(hidden, generator=g) * 0.1).to(wd)
    out = torch.empty(19, hidden, dtype=od, device=DEV)
    kernels.rmsnorm(x.to(DEV), w.to(DEV), 1e-5, 1.0, out)
    close(out, plain.rms_norm(x, w, 1e-5), od)
    rows = torch.tensor([18, 0, 7], dtype=torch.int32)
    out2 = torch.empty(3, hidden, dtype=od, device=DEV)
    kernels.rmsnorm(x.to(DEV), w.to(DEV), 1e-5, 1.0, out2, rows.to(DEV))
    close(out2, plain.rms_norm(x[rows.long()], w, 1e-5), od)


@pytest.mark.parametrize("yd,wd,od", [(torch.float32, torch.float32, torch.float32),
                                       (torch.float32, torch.bfloat16, torch.bfloat16),
                                       (torch.bfloat16, torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("post,nxt", [(True, True), (True, False), (False, True), (False, False)])
def test_residual_rmsnorm(yd, wd, od, post, nxt):
    hidden = 328
    g = torch.Generator().manual_seed(2)
    h = torch.randn(11, hidden, generator=g) * 5
    y = (torch.randn(11, hidden, generator=g) * 2).to(yd)
    w1 = (torch.randn(hidden, generator=g) * 0.1).to(wd)
    w2 = (torch.randn(hidden, generator=g) * 0.1).to(wd)
    hd = h.clone().to(DEV)
    out = torch.empty(11, hidden, dtype=od, device=DEV) if nxt else None
    kernels.residual_rmsnorm(hd, y.to(DEV), w1.to(DEV) if post else None, 1e-6, 1.0,
                             w2.to(DEV) if nxt else None, 1e-5, 1.0, out)
    h_ref = h.double() + (plain.rms_norm(y, w1, 1e-6) if post else y.double())
    close(hd, h_ref, torch.float32)
    if nxt:
        close(out, plain.rms_norm(h_ref, w2, 1e-5), od)


@pytest.mark.parametrize("rows,hidden", [(1500, 2304), (2000, 328), (1300, 3584), (1185, 1024), (5000, 2304)])
@pytest.mark.parametrize("post,nxt", [(True, True), (False, True), (True, False)])
def test_residual_rmsnorm_of_a_prompts_rows(rows, hidden, post, nxt):
    """Thousands of rows (a prompt): the form with the row in shared memory, at one and at several rounds of
    its blocks and at widths of one to four chunks per thread."""
    g = torch.Generator().manual_seed(rows + hidden)
    h = torch.randn(rows, hidden, generator=g) * 5
    y = (torch.randn(rows, hidden, generator=g) * 2).to(torch.bfloat16)
    w1 = (torch.randn(hidden, generator=g) * 0.1).to(torch.bfloat16)
    w2 = (torch.randn(hidden, generator=g) * 0.1).to(torch.bfloat16)
    hd = h.clone().to(DEV)
    out = torch.full((rows, hidden), float("nan"), dtype=torch.bfloat16, device=DEV) if nxt else None
    kernels.residual_rmsnorm(hd, y.to(DEV), w1.to(DEV) if post else None, 1e-6, 1.0,
                             w2.to(DEV) if nxt else None, 1e-5, 1.0, out)
    h_ref = h.double() + (plain.rms_norm(y, w1, 1e-6) if post else y.double())
    close(hd, h_ref, torch.float32)
    if nxt:
        close(out, plain.rms_norm(h_ref, w2, 1e-5), torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("act", ["gelu_tanh", "silu"])
def test_gated_act(dtype, act):
    g = torch.Generator().manual_seed(3)
    gu = (torch.randn(7, 2 * 330, generator=g) * 3).to(dtype)
    out = torch.empty(7, 330, dtype=dtype, device=DEV)
    kernels.gated_act(gu.to(DEV), out, act)
    gate, up = gu[:, :330].double(), gu[:, 330:].double()
    ref = (plain.gelu_tanh(gate) if act == "gelu_tanh" else gate * torch.sigmoid(gate)) * up
    close(out, ref, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_softcap(dtype):
    g = torch.Generator().manual_seed(4)
    x = (torch.randn(3, 1001, generator=g) * 40).to(dtype)
    out = torch.empty(3, 1001, dtype=torch.float32, device=DEV)
    kernels.softcap(x.to(DEV), out, 30.0)
    close(out, plain.soft_cap(x.double(), 30.0), torch.float32)
    assert float(out.abs().max()) <= 30.0
    kernels.softcap(x.to(DEV), out, 0.0)
    close(out, x.double(), torch.float32)


@pytest.mark.parametrize("M,N,K", [(1, 7, 5), (3, 130, 96), (65, 200, 330), (128, 64, 16), (17, 1000, 203)])
def test_linear_f32(M, N, K):
    g = torch.Generator().manual_seed(5)
    x = torch.randn(M, K, generator=g)
    w = torch.randn(N, K, generator=g)
    out = torch.empty(M, N, dtype=torch.float32, device=DEV)
    kernels.linear_f32(x.to(DEV), w.to(DEV), out)
    close(out, plain.linear(x, w), torch.float32)
    # a row gives the same bits alone and in the batch
    one = torch.empty(1, N, dtype=torch.float32, device=DEV)
    kernels.linear_f32(x[M - 1:M].to(DEV), w.to(DEV), one)
    assert torch.equal(one[0], out[M - 1])


@pytest.mark.parametrize("M", [1, 2, 5, 16, 17, 33, 70])
@pytest.mark.parametrize("N,K", [(8, 4), (33, 516), (2304, 2304), (136, 9216), (4750, 1028), (9500, 512)])
def test_linear_f32_kernels_and_cuts(M, N, K):
    """Streams of 8, 16 and 32 rows a block, tiles of 32 and 64 rows, cut along K and not: float sums, one order."""
    g = torch.Generator(device=DEV).manual_seed(M * N + K)
    x = torch.randn(M, K, generator=g, device=DEV)
    w = torch.randn(N, K, generator=g, device=DEV)
    out = torch.full((M, N), float("nan"), device=DEV)
    kernels.linear_f32(x, w, out)
    ref = x.double() @ w.double().T
    # chains of at most 256 fmas, then their sums: each rounding is at most 2^-24 of a partial sum
    bound = (256 + K / 256) * 2.0 ** -24 * (x.abs().double() @ w.abs().double().T)
    assert bool(((out.double() - ref).abs() <= bound).all())
    one = torch.empty(1, N, device=DEV)
    kernels.linear_f32(x[M - 1:], w, one)
    assert torch.equal(one[0], out[M - 1])
    # the same numbers off the 16-byte boundaries: the kernel for any operands, in the same order
    wide = torch.empty(M, K + 1, device=DEV)
    wide[:, 1:] = x
    again = torch.empty(M, N, device=DEV)
    kernels.linear_f32(wide[:, 1:], w, again)
    assert torch.equal(again, out)


@pytest.mark.parametrize("M", [1, 2, 5, 16, 17, 33, 70])
@pytest.mark.parametrize("N,K", [(300, 3072), (112, 9216), (1000, 1028), (2040, 512), (5000, 204)])
def test_linear_f32_kernels_and_cuts_of_weights_for_cuda_cores(M, N, K):
    """The same of weights that are all too small for tensor cores."""
    assert not kernels.linear_f32_tc_ok(torch.empty(N, K, device=DEV))
    test_linear_f32_kernels_and_cuts(M, N, K)


@pytest.mark.parametrize("M", [1, 8, 16, 31, 33, 64, 100])
@pytest.mark.parametrize("N,K", [(5, 4), (128, 16), (130, 100), (257, 1540), (96, 3072)])
def test_linear_f32_every_kernel_gives_the_same_bits(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N * K)
    x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
    ref = torch.empty(M, N, device=DEV)
    kernels._linear_f32(x, w, ref, 0, 0)
    segs = -(-K // kernels.F32_SEGMENT)
    for kind, cut in [(k, c) for k in (1, 32, 64) for c in range(segs if k > 1 else 1) if k > 1 or M <= 16]:
        out = torch.full((M, N), float("nan"), device=DEV)
        kernels._linear_f32(x, w, out, kind, cut)
        assert torch.equal(out, ref), (kind, cut)


@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 160, 161, 330])
@pytest.mark.parametrize("N,K", [(4100, 260), (1024, 1028), (130, 9216), (20000, 256)])
def test_linear_f32_on_tensor_cores(M, N, K):
    """One, two, four and eight slices of K, ends of K and of the rows inside a tile, every width of the token tile."""
    assert kernels.linear_f32_tc_slices(N, K) == {4100: 2, 1024: 4, 130: 8, 20000: 1}[N]
    g = torch.Generator(device=DEV).manual_seed(M * N + K)
    x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
    x[:, ::3] *= 1e-3                                        # (rows whose numbers differ widely)
    wide = torch.full((M, N + 3), float("nan"), device=DEV)
    kernels.linear_f32(x, w, wide[:, :N])
    out = wide[:, :N]
    assert kernels.linear_f32_tc_status(reset=True) == 0 and bool(wide[:, N:].isnan().all())
    ref = x.double() @ w.double().T
    # a product 3 * 2^-24; per 64 k twelve steps of the tensor core, each good to 2^-22 of what it adds; K / 64 float additions;
    # what is too small for its row's scale 2^-38 of its largest
    size = x.abs().double() @ w.abs().double().T
    least = 2.0 ** -38 * K * x.abs().amax(1, keepdim=True).double() * w.abs().amax(1).double()
    assert bool(((out.double() - ref).abs() <= (3 + 48 + K / 64) * 2.0 ** -24 * size + least).all())
    plain_sums = torch.empty(M, N, device=DEV)
    kernels._linear_f32(x, w, plain_sums, 0, 0)
    assert float((out.double() - ref).norm()) <= 1.05 * float((plain_sums.double() - ref).norm())     # no less precise
    for m in (0, M - 1):                                     # alone, and off the 16-byte boundaries
        row = torch.empty(1, K + 1, device=DEV)
        row[:, 1:] = x[m]
        one = torch.empty(1, N, device=DEV)
        kernels.linear_f32(row[:, 1:], w, one)
        assert torch.equal(one[0], out[m])


def tc_f32_bound(K):
    """Of the float product on tensor cores, as a share of sum |x w|: a product good to 2^-24; for 64 k four steps of the tensor
    core with the large parts, each good to 2^-22 of what it adds, and twenty with parts 2^-8 as large; K / 64 float additions."""
    return (1 + 4 * 4 + 1 + K / 64) * 2.0 ** -24


@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 160, 161, 330])
@pytest.mark.parametrize("N,K", [(4100, 260), (1024, 1028), (130, 9216), (20000, 256)])
def test_linear_f32_on_tensor_cores_of_whole_floats(M, N, K):
    """Every sum to what three parts a float allow: nothing for a row's largest number."""
    assert kernels.linear_f32_tc_slices(N, K) > 0
    g = torch.Generator(device=DEV).manual_seed(M * N + K)
    x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
    x[:, ::3] *= 1e-3
    out = torch.full((M, N), float("nan"), device=DEV)
    kernels.linear_f32(x, w, out)
    size = x.abs().double() @ w.abs().double().T
    assert bool(((out.double() - x.double() @ w.double().T).abs() <= tc_f32_bound(K) * size).all())


@pytest.mark.parametrize("beside", [1e4, 1e8, 1e12, 2.0 ** 40, 1e30])
@pytest.mark.parametrize("M,off", [(3, 0), (3, 1), (20, 0), (40, 0), (40, 1), (300, 0)])
@pytest.mark.parametrize("where", ["x", "w"])
def test_linear_f32_keeps_numbers_beside_much_larger_ones(where, M, off, beside):
    """A large number in every 64 k that meets a zero: the others' sum is as good as without it."""
    N, K = 2052, 520
    assert kernels.linear_f32_tc_slices(N, K) > 1
    g = torch.Generator(device=DEV).manual_seed(M + off)
    x, w = torch.randn(M, K + off, generator=g, device=DEV)[:, off:], torch.randn(N, K, generator=g, device=DEV)
    big, zero = (x, w) if where == "x" else (w, x)
    big[:, 5::64] *= beside
    zero[:, 5::64] = 0.0
    assert kernels.linear_f32_tc_ok(w)
    out = torch.empty(M, N, device=DEV)
    kernels.linear_f32(x, w, out)
    error = (out.double() - x.double() @ w.double().T).abs()
    assert bool((error <= tc_f32_bound(K) * (x.abs().double() @ w.abs().double().T)).all())
    gated, both = torch.empty(M, N // 2, device=DEV), torch.empty(M, N // 2, device=DEV)
    kernels.linear_f32_gated(x, w, gated, "silu")
    kernels.gated_act(out, both, "silu")
    assert torch.equal(gated, both)


@pytest.mark.parametrize("M", [1, 20, 40, 200])
def test_linear_f32_on_tensor_cores_at_the_ends_of_the_range(M):
    """Numbers of which three parts do not hold all bits, beside others that make a sum of ordinary size of them; sums whose
    terms all end below the smallest normal number; an identity returns x."""
    N, K = 2048, 640
    g = torch.Generator(device=DEV).manual_seed(M)
    x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
    x[:, 7] *= 2.0 ** -118
    w[:, 7] *= 2.0 ** 110
    x[:, 8:] *= 2.0 ** -20
    w[::2, 7] *= 2.0 ** 7 - 1
    w[1::4, :7], w[1::4, 8:] = 0.0, 0.0                      # rows with nothing but that number
    w[3::8, 8:] *= 2.0 ** -118
    x[0, 8:] = 0.0
    out = torch.empty(M, N, device=DEV)
    kernels.linear_f32(x, w, out)
    error = (out.double() - x.double() @ w.double().T).abs()
    assert bool((error <= tc_f32_bound(K) * (x.abs().double() @ w.abs().double().T) + K * 2.0 ** -149).all())
    x, w = torch.randn(M, K, generator=g, device=DEV) * 2.0 ** -66, torch.randn(N, K, generator=g, device=DEV) * 2.0 ** -72
    kernels.linear_f32(x, w, out)
    error = (out.double() - x.double() @ w.double().T).abs()
    assert bool((error <= tc_f32_bound(K) * (x.abs().double() @ w.abs().double().T) + K * 2.0 ** -149).all())
    x, w = torch.randn(M, 1024, generator=g, device=DEV), torch.eye(1024, device=DEV)
    x[:, ::3] *= 1e9
    out = torch.empty(M, 1024, device=DEV)
    kernels.linear_f32(x, w, out)
    assert kernels.linear_f32_tc_ok(w) and torch.equal(out, x)


@pytest.mark.parametrize("M,off", [(3, 0), (20, 1), (40, 0), (40, 1), (200, 0)])
@pytest.mark.parametrize("low,high,zeros", [(-120, 60, 0.0), (-126, -20, 0.2), (-60, 58, 0.2), (20, 58, 0.0), (-110, -50, 0.9)])
def test_linear_f32_on_tensor_cores_of_numbers_of_all_sizes(M, off, low, high, zeros):
    """Every number with an exponent of its own, some of them zeros (up to 2^60: products of 2^126 would run over)."""
    N, K = 2052, 520
    g = torch.Generator(device=DEV).manual_seed(M + off - low)

    def draw(*shape):
        t = torch.randn(*shape, generator=g, device=DEV) * torch.exp2(torch.empty(*shape, device=DEV).uniform_(low, high, generator=g))
        t[torch.rand(*shape, generator=g, device=DEV) < zeros] = 0.0
        return t
    x, w = draw(M, K + off)[:, off:], draw(N, K)
    out = torch.empty(M, N, device=DEV)
    kernels.linear_f32(x, w, out)
    error = (out.double() - x.double() @ w.double().T).abs()
    assert bool((error <= tc_f32_bound(K) * (x.abs().double() @ w.abs().double().T) + K * 2.0 ** -149).all())


@pytest.mark.parametrize("M", [3, 20, 40, 300])
@pytest.mark.parametrize("N,K", [(2052, 520), (20000, 260), (2304, 2304)])
def test_linear_f32_on_tensor_cores_of_nan(M, N, K):
    """A NaN of a token or of a row of W is in all its sums and in no other."""
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
    before, out = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    kernels.linear_f32(x, w, before)
    x[M - 1, K - 1], w[5, 0] = torch.nan, torch.nan
    w[6, 3] = torch.inf
    kernels.linear_f32(x, w, out)
    nan = torch.zeros(M, N, dtype=torch.bool, device=DEV)
    nan[M - 1], nan[:, 5] = True, True
    assert torch.equal(out.isnan(), nan)
    keep = torch.ones(M, N, dtype=torch.bool, device=DEV)
    keep[M - 1], keep[:, 5:7] = False, False
    assert torch.equal(out[keep], before[keep]) and bool(out[:-1, 6].isinf().all())


@pytest.mark.parametrize("kind", ["normal", "positive", "spread"])
@pytest.mark.parametrize("M,N,K", [(3, 4096, 2304), (300, 2304, 9216)])
def test_linear_f32_on_tensor_cores_is_no_less_precise_than_fmas(kind, M, N, K):
    g = torch.Generator(device=DEV).manual_seed(5)
    x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV) * 0.02
    if kind == "positive":
        x, w = x.abs(), w.abs()
    if kind == "spread":
        x, w = x * torch.exp(3 * torch.randn(M, K, generator=g, device=DEV)), w * torch.exp(2 * torch.randn(N, K, generator=g, device=DEV))
    out, fmas = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    kernels.linear_f32(x, w, out)
    kernels._linear_f32(x, w, fmas, 0, 0)
    ref, size = x.double() @ w.double().T, x.abs().double() @ w.abs().double().T
    # sums of one sign: the tensor core cuts off half a last place at each of four steps, with a quarter to the whole of 64 k's sum
    cut = 1.8 * 2.0 ** -24 * float(ref.norm()) if kind == "positive" else 0.0
    assert float((out.double() - ref).norm()) <= float((fmas.double() - ref).norm()) + cut
    assert float(((out.double() - ref).abs() / size).max()) <= float(((fmas.double() - ref).abs() / size).max())


def test_linear_f32_of_weights_that_the_kernel_before_it_made():
    """More than 16 rows: the weights are read behind the kernel before."""
    g = torch.Generator(device=DEV).manual_seed(3)
    made = torch.randn(4096, 2304, generator=g, device=DEV).to(torch.bfloat16)
    for M in (17, 40, 200):
        x, out = torch.randn(M, 2304, generator=g, device=DEV), torch.empty(M, 4096, device=DEV)
        want = torch.empty(M, 4096, device=DEV)
        kernels.linear_f32(x, made.float(), want)
        for _ in range(5):
            w = torch.full((4096, 2304), float("nan"), device=DEV)
            torch.cuda.synchronize()
            kernels.cast(made, w)
            kernels.linear_f32(x, w, out)
            assert torch.equal(out, want)
            kernels.linear_f32(x, w, out, standing=True)
            assert torch.equal(out, want)


def test_linear_f32_on_tensor_cores_of_infinities_and_the_smallest_numbers():
    """What a sum of parts cannot say is said by the floats themselves; the rows beside keep their bits."""
    g = torch.Generator(device=DEV).manual_seed(12)
    M, N, K = 40, 2048, 520
    x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
    w[7, :] = w[7, :].to(torch.bfloat16).float()
    before = torch.empty(M, N, device=DEV)
    kernels.linear_f32(x, w, before)
    x[3, 5], x[4, 77], x[5, 519], x[6, :4] = torch.inf, -torch.inf, torch.nan, 3.4e38
    x[8] *= 1e-35
    x[9] *= 1e30
    w[9, 1], w[11] = torch.inf, 0.0
    w[12] *= 1e-36
    w[13] *= 1e-30
    out, plain_sums = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    kernels.linear_f32(x, w, out)
    kernels._linear_f32(x, w, plain_sums, 0, 0)
    others = torch.arange(M, device=DEV) != 6               # (sums of the largest numbers run over on their way, or do not)
    for same in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(same(out[others]), same(plain_sums[others]))
    ref, size = x.double() @ w.double().T, x.abs().double() @ w.abs().double().T
    ok = ref.isfinite() & plain_sums.isfinite() & out.isfinite()
    bound = 512 * 2.0 ** -24 * size + K * 2.0 ** -149
    assert bool((((out.double() - ref).abs() <= bound) | ~ok).all())
    rows = torch.tensor([m for m in range(M) if m not in (3, 4, 5, 6, 8, 9)], device=DEV)
    cols = torch.tensor([n for n in range(N) if n not in (9, 11, 12, 13)], device=DEV)
    assert torch.equal(out[rows][:, cols], before[rows][:, cols])


@pytest.mark.parametrize("M", [1, 16, 17, 32])
@pytest.mark.parametrize("N,K", [(4100, 260), (2050, 1028), (136, 9216)])
def test_linear_f32_in_slices(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x, w = torch.randn(M, K + 1, generator=g, device=DEV)[:, 1:], torch.randn(N, K, generator=g, device=DEV)
    x[0, 3], w[5] = torch.nan, w[5] * 1e-36
    n = kernels.linear_f32_parts(x, w)
    assert n == kernels.linear_f32_tc_slices(N, K) > 1 and kernels.linear_f32_parts(x.repeat(33, 1), w) == 1
    sums, out = torch.full((n, M, N), 7.0, device=DEV), torch.empty(M, N, device=DEV)
    kernels.linear_f32_slices_into(x, w, sums)
    kernels.linear_f32(x, w, out)
    total = sums[0].clone()
    for s in sums[1:]:
        total += s
    assert torch.equal(total.nan_to_num(7.0), out.nan_to_num(7.0))


@pytest.mark.parametrize("activation,limit", [("gelu_tanh", 0.0), ("silu", 0.0), ("clamped_gate", 1.5)])
@pytest.mark.parametrize("M,F,K", [(1, 2048, 256), (16, 520, 1028), (33, 9472, 256), (170, 2100, 512)])
def test_linear_f32_gated(M, F, K, activation, limit):
    g = torch.Generator(device=DEV).manual_seed(M + F)
    x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(2 * F, K, generator=g, device=DEV) / K ** 0.5
    w[1, 3] = torch.inf
    both, want, out = torch.empty(M, 2 * F, device=DEV), torch.empty(M, F, device=DEV), torch.empty(M, F, device=DEV)
    kernels.linear_f32(x, w, both)
    kernels.gated_act(both, want, activation, limit)
    kernels.linear_f32_gated(x, w, out, activation, limit)
    assert torch.equal(out.nan_to_num(7.0), want.nan_to_num(7.0))


@pytest.mark.parametrize("T,n_kv", [(1280, 4), (2048, 4)])
def test_prompt_attention_cut_in_halves_repeats_itself(T, n_kv):
    """Which half of a row block comes second and merges is a matter of time; the bits are not."""
    group, hd = 2, 256
    assert kernels.attention_prefill_tc_split(T, n_kv, group, 0, 1) > 0
    g = torch.Generator(device=DEV).manual_seed(T)
    qkv = torch.randn(T, (n_kv * group + 2 * n_kv) * hd, generator=g, device=DEV).to(torch.bfloat16)
    cu, q = torch.tensor([0, T], dtype=torch.int32, device=DEV), n_kv * group * hd
    noise = torch.empty(64 << 20, device=DEV)
    outs = []
    for i in range(24):
        if i % 2:
            noise.normal_()                                   # (other blocks on the SMs as the launch begins)
        outs.append(torch.empty(T, q, dtype=torch.bfloat16, device=DEV))
        kernels.attention_prefill_tc(qkv[:, :q], outs[-1], cu, qkv[:, q:q + n_kv * hd], qkv[:, q + n_kv * hd:], n_kv=n_kv, group=group,
                                     head_dim=hd, scale=hd ** -0.5, cap=50.0, window=0, batch=1, max_q_len=T)
    assert all(torch.equal(o, outs[0]) for o in outs[1:])


def test_linear_f32_takes_no_scratch_for_operands_it_does_not_cut():
    x = torch.zeros(300, 2305, device=DEV)[:, 1:]
    w, out = torch.zeros(2304, 2304, device=DEV), torch.empty(300, 2304, device=DEV)
    assert kernels.linear_f32_plan(300, 2304, 2304, kernels.device_sms())[1] > 0
    kernels.linear_f32(x, w, out)
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    kernels.linear_f32(x, w, out)
    assert torch.cuda.max_memory_allocated() == before


def test_linear_f32_takes_no_scratch_for_small_operands_it_does_not_cut():
    x = torch.zeros(300, 3073, device=DEV)[:, 1:]
    w, out = torch.zeros(300, 3072, device=DEV), torch.empty(300, 300, device=DEV)
    assert not kernels.linear_f32_tc_ok(w) and kernels.linear_f32_plan(300, 300, 3072, kernels.device_sms())[1] > 0
    kernels.linear_f32(x, w, out)
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    kernels.linear_f32(x, w, out)
    assert torch.cuda.max_memory_allocated() == before


def test_linear_f32_strided_views():
    g = torch.Generator().manual_seed(6)
    big = torch.randn(9, 3 * 48, generator=g).to(DEV)
    w = torch.randn(20, 48, generator=g).to(DEV)
    out = torch.zeros(9, 64, dtype=torch.float32, device=DEV)
    kernels.linear_f32(big[:, 48:96], w, out[:, 8:28])
    close(out[:, 8:28], plain.linear(big[:, 48:96].cpu(), w.cpu()), torch.float32)
    assert float(out[:, :8].abs().max()) == 0 and float(out[:, 28:].abs().max()) == 0


@pytest.mark.parametrize("M", [1, 3, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(16, 64), (40, 72), (1000, 200), (2304, 2304), (48, 9216)])
def test_skinny_gemm(M, N, K):
    g = torch.Generator().manual_seed(M * 1000 + N + K)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g) * 0.1).to(torch.bfloat16)
    ref = plain.linear(x, w)
    for dt in (torch.bfloat16, torch.float32):
        out = torch.full((M, N), 7.0, dtype=dt, device=DEV)
        kernels.skinny_gemm(x.to(DEV), w.to(DEV), out)
        close(out, ref, torch.float32 if dt == torch.float32 else torch.bfloat16,
              scale=float(ref.abs().max()) * (50 if dt == torch.float32 else 1))
    out = torch.empty(M, N, dtype=torch.float32, device=DEV)
    kernels.skinny_gemm(x.to(DEV), w.to(DEV), out, "softcap", cap=3.0)
    close(out, plain.soft_cap(ref, 3.0), torch.float32, scale=3.0 * 50)
    # a row gives the same bits alone and in the batch
    one = torch.empty(1, N, dtype=torch.float32, device=DEV)
    kernels.skinny_gemm(x[M - 1:M].to(DEV), w.to(DEV), one, "softcap", cap=3.0)
    assert torch.equal(one[0], out[M - 1])


@pytest.mark.parametrize("M,F,K,act", [(1, 16, 64, "gelu_tanh"), (8, 328, 96, "silu"), (13, 9216, 128, "gelu_tanh"),
                                       (16, 40, 2304, "gelu_tanh")])
def test_skinny_gemm_gated(M, F, K, act):
    g = torch.Generator().manual_seed(F + K)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(2 * F, K, generator=g) * 0.1).to(torch.bfloat16)
    gate, up = plain.linear(x, w[:F]), plain.linear(x, w[F:])
    ref = (plain.gelu_tanh(gate) if act == "gelu_tanh" else gate * torch.sigmoid(gate)) * up
    out = torch.empty(M, F, dtype=torch.bfloat16, device=DEV)
    kernels.skinny_gemm(x.to(DEV), w.to(DEV), out, "gated", act)
    close(out, ref, torch.bfloat16)


@pytest.mark.parametrize("parts", [2, 3, 8])
def test_skinny_gemm_partial_sums_feed_the_residual_kernel(parts):
    g = torch.Generator().manual_seed(parts)
    M, N, K = 5, 328, 9216
    x = torch.randn(M, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g) * 0.05).to(torch.bfloat16)
    y = torch.full((parts, M, N), float("nan"), dtype=torch.float32, device=DEV)
    kernels.skinny_gemm(x.to(DEV), w.to(DEV), y)
    ref = plain.linear(x, w)
    close(y.sum(0), ref, torch.float32, scale=float(ref.abs().max()) * 50)
    h = torch.randn(M, N, generator=g)
    gain = (torch.randn(N, generator=g) * 0.1).to(torch.bfloat16)
    hd_ = h.clone().to(DEV)
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    kernels.residual_rmsnorm(hd_, y, gain.to(DEV), 1e-6, 1.0, gain.to(DEV), 1e-6, 1.0, out)
    h_ref = h.double() + plain.rms_norm(ref, gain, 1e-6)
    close(hd_, h_ref, torch.float32, scale=float(h_ref.abs().max()) * 50)
    close(out, plain.rms_norm(h_ref, gain, 1e-6), torch.bfloat16)
    assert kernels.skinny_parts(torch.empty(8, 9216), torch.empty(2304, 9216), sms=148) == 3
    assert kernels.skinny_parts(torch.empty(8, 2304), torch.empty(18432, 2304)) == 1


@pytest.mark.parametrize("pairs", [True, False])
@pytest.mark.parametrize("M,N,K", [(17, 256, 64), (128, 256, 256), (100, 300, 200), (333, 2304, 2048), (1000, 40, 72),
                                   (2048, 512, 9216), (257, 520, 136)])
def test_gemm_tc(M, N, K, pairs):
    """One block per 128 x 256 tile, and a pair of SMs per 256 x 256 tile (cta_group::2)."""
    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g) * 0.05).to(torch.bfloat16)
    ref = plain.linear(x, w)
    for dt in (torch.bfloat16, torch.float32):
        out = torch.full((M, N), 7.0, dtype=dt, device=DEV)
        kernels.gemm_tc(x.to(DEV), w.to(DEV), out, pairs=pairs)
        close(out, ref, dt, scale=float(ref.abs().max()) * (50 if dt == torch.float32 else 1))
    assert kernels.gemm_tc_status() == 0


@pytest.mark.parametrize("pairs", [True, False])
@pytest.mark.parametrize("M,F,K,act", [(17, 128, 64, "gelu_tanh"), (300, 384, 200, "silu"), (2048, 9216, 2304, "gelu_tanh")])
def test_gemm_tc_gated(M, F, K, act, pairs):
    g = torch.Generator().manual_seed(F + K)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(2 * F, K, generator=g) * 0.05).to(torch.bfloat16)
    xd, wd = x.to(DEV), w.to(DEV)
    out = torch.empty(M, F, dtype=torch.bfloat16, device=DEV)
    kernels.gemm_tc(xd, wd, out, "gated", act, pairs=pairs)
    gate, up = xd.double() @ wd[:F].double().t(), xd.double() @ wd[F:].double().t()      # float64 on the device: fast
    ref = (plain.gelu_tanh(gate) if act == "gelu_tanh" else gate * torch.sigmoid(gate)) * up
    close(out, ref, torch.bfloat16)
    assert kernels.gemm_tc_status() == 0


@pytest.mark.parametrize("M,N,K,parts", [(1, 128, 256, 1), (8, 2304, 2048, 8), (16, 300, 200, 1), (17, 4096, 2304, 1),
                                         (64, 2304, 9216, 8), (128, 512, 512, 3), (33, 1000, 72, 1)])
def test_gemm_stream(M, N, K, parts):
    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(N, K, generator=g) * 0.05).to(torch.bfloat16).to(DEV)
    ref = x.double() @ w.double().t()
    for dt in (torch.bfloat16, torch.float32):
        out = torch.full((M, N), 7.0, dtype=dt, device=DEV)
        kernels.gemm_stream(x, w, out)
        close(out, ref, dt, scale=float(ref.abs().max()) * (50 if dt == torch.float32 else 1))
    if parts > 1:
        nkb = (K + 63) // 64
        per = (nkb + parts - 1) // parts
        parts = (nkb + per - 1) // per                      # no empty slice
        y = torch.full((parts, M, N), float("nan"), dtype=torch.float32, device=DEV)
        kernels.gemm_stream(x, w, y)
        close(y.sum(0), ref, torch.float32, scale=float(ref.abs().max()) * 50)
    out = torch.empty(M, N, dtype=torch.float32, device=DEV)
    kernels.gemm_stream(x, w, out, "softcap", cap=3.0)
    close(out, plain.soft_cap(ref, 3.0), torch.float32, scale=3.0 * 50)
    assert kernels.gemm_stream_status() == 0


@pytest.mark.parametrize("M,F,K,act", [(1, 64, 64, "gelu_tanh"), (8, 9216, 2304, "gelu_tanh"), (50, 128, 72, "silu"),
                                       (100, 320, 128, "gelu_tanh")])
def test_gemm_stream_gated(M, F, K, act):
    g = torch.Generator().manual_seed(F + K)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(2 * F, K, generator=g) * 0.05).to(torch.bfloat16).to(DEV)
    out = torch.empty(M, F, dtype=torch.bfloat16, device=DEV)
    kernels.gemm_stream(x, w, out, "gated", act)
    gate, up = x.double() @ w[:F].double().t(), x.double() @ w[F:].double().t()
    ref = (plain.gelu_tanh(gate) if act == "gelu_tanh" else gate * torch.sigmoid(gate)) * up
    close(out, ref, torch.bfloat16)
    assert kernels.gemm_stream_status() == 0
    # o of Gemma 2 2B (32 blocks of K, 18 row tiles): a ring's worth of K per item, four slices
    assert kernels.gemm_stream_parts(torch.empty(8, 2048), torch.empty(2304, 2048)) == 4
    assert kernels.gemm_stream_parts(torch.empty(8, 9216), torch.empty(2304, 9216)) == 8
    assert kernels.gemm_stream_parts(torch.empty(8, 2304), torch.empty(256000, 2304)) == 1


@pytest.mark.parametrize("M", [1, 16, 17, 33, 128])
@pytest.mark.parametrize("kind,N,K", [("store", 128 * 150 - 40, 72), ("store", 128 * 310 + 8, 200), ("parts", 1000, 64 * 44),
                                      ("gated", 64 * 150, 72), ("gated", 64 * 300, 392)])
def test_gemm_stream_with_two_blocks_an_sm(M, kind, N, K):
    """More items than SMs: one round of two blocks an SM, and more than a round; remainders of rows and of K."""
    g = torch.Generator(device=DEV).manual_seed(N + M)
    x = torch.randn(M, K, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(2 * N if kind == "gated" else N, K, generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    ref = x.double() @ w.double().t()
    if kind == "gated":
        out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
        kernels.gemm_stream(x, w, out, "gated", "gelu_tanh")
        close(out, plain.gelu_tanh(ref[:, :N]) * ref[:, N:], torch.bfloat16)
    else:
        out = torch.empty((22, M, N) if kind == "parts" else (M, N), dtype=torch.float32, device=DEV)
        kernels.gemm_stream(x, w, out)
        close(out.sum(0) if kind == "parts" else out, ref, torch.float32, scale=float(ref.abs().max()) * 50)
    assert kernels.gemm_stream_status() == 0


def test_gemm_tc_strided_views():
    g = torch.Generator().manual_seed(2)
    big = torch.randn(40, 3 * 64, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(24, 64, generator=g).to(torch.bfloat16).to(DEV)
    x = big[:, 64:128]
    assert kernels.gemm_tc_ok(x, w, sms=1) and not kernels.gemm_tc_ok(big[:, 1:65], w, sms=1)
    assert not kernels.gemm_tc_ok(x, w)            # one tile only: not worth a persistent kernel
    wide = torch.zeros(40, 64, dtype=torch.float32, device=DEV)
    kernels.gemm_tc(x, w, wide[:, 8:32])
    close(wide[:, 8:32], plain.linear(x.cpu(), w.cpu()), torch.float32, scale=float(wide.abs().max()) * 50)
    assert float(wide[:, :8].abs().max()) == 0 and float(wide[:, 32:].abs().max()) == 0


def test_skinny_gemm_strided_input():
    g = torch.Generator().manual_seed(1)
    big = torch.randn(5, 3 * 64, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(24, 64, generator=g).to(torch.bfloat16).to(DEV)
    x = big[:, 64:128]
    assert kernels.skinny_ok(x, w) and not kernels.skinny_ok(big[:, 1:65], w)
    out = torch.empty(5, 24, dtype=torch.float32, device=DEV)
    kernels.skinny_gemm(x, w, out)
    close(out, plain.linear(x.cpu(), w.cpu()), torch.float32, scale=float(out.abs().max()) * 50)


def _rope_case(dtype, n_q, n_kv, hd, ring, page, lengths, seed):
    """Prompt pass of unequal sequences: rotation against the oracle and the pages written."""
    g = torch.Generator().manual_seed(seed)
    B = len(lengths)
    T = sum(lengths)
    width = (n_q + 2 * n_kv) * hd
    qkv = torch.randn(T, width, generator=g).to(dtype)
    positions = torch.cat([torch.arange(n) for n in lengths]).int()
    theta = 1000.0
    half = hd // 2
    inv = torch.tensor(theta, dtype=torch.float64) ** (-2.0 * torch.arange(half, dtype=torch.float64) / hd)
    ang = torch.arange(max(lengths), dtype=torch.float64)[:, None] * inv[None]
    table = torch.stack([ang.cos(), ang.sin()], -1).float()
    pages_per = [min((n + page - 1) // page, ring // page) for n in lengths]
    n_pages = sum(pages_per) + 3
    perm = torch.randperm(n_pages, generator=g).tolist()        # scattered page ids
    pt = torch.zeros(B, max(pages_per), dtype=torch.int32)
    it = iter(perm)
    for b in range(B):
        for j in range(pages_per[b]):
            pt[b, j] = next(it)
    kp = torch.zeros(n_pages, n_kv, page, hd, dtype=dtype, device=DEV)
    vp = torch.zeros_like(kp)
    dq = qkv.clone().to(DEV)
    rows = []
    for b, n in enumerate(lengths):
        for p_ in range(n):
            ridx = p_ % ring
            rows.append(int(pt[b, ridx // page]) * page + ridx % page if p_ >= n - ring else -1)
    kernels.rope_kv_write(dq, positions.to(DEV), table.to(DEV), n_q, n_kv, hd, hd, kp, vp,
                          torch.tensor(rows, dtype=torch.int32, device=DEV), page)
    q_ref = plain.rope(qkv[:, :n_q * hd], positions, hd, theta)
    k_ref = plain.rope(qkv[:, n_q * hd:(n_q + n_kv) * hd], positions, hd, theta)
    close(dq[:, :n_q * hd], q_ref, dtype)
    close(dq[:, n_q * hd:(n_q + n_kv) * hd], k_ref, dtype)
    assert torch.equal(dq[:, (n_q + n_kv) * hd:].cpu(), qkv[:, (n_q + n_kv) * hd:])
    kp, vp, dq = kp.cpu(), vp.cpu(), dq.cpu()
    t = 0
    for b, n in enumerate(lengths):
        for p in range(n):
            if p >= n - ring:
                ridx = p % ring
                pg = int(pt[b, ridx // page])
                assert torch.equal(kp[pg, :, ridx % page, :].reshape(-1), dq[t, n_q * hd:(n_q + n_kv) * hd]), (b, p)
                assert torch.equal(vp[pg, :, ridx % page, :].reshape(-1), dq[t, (n_q + n_kv) * hd:]), (b, p)
            t += 1


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rope_kv_write_all_keys(dtype):
    _rope_case(dtype, n_q=6, n_kv=3, hd=48, ring=1 << 30, page=64, lengths=[1, 70, 130], seed=7)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rope_kv_write_ring(dtype):
    # prompts longer than the ring: only the last `ring` places are written, each exactly once
    _rope_case(dtype, n_q=2, n_kv=1, hd=32, ring=64, page=32, lengths=[200, 64, 65, 3], seed=8)


@pytest.mark.parametrize("n_q,n_kv,hd,slices", [(8, 4, 256, 4), (6, 1, 32, 1), (3, 3, 48, 3), (32, 16, 128, 2)])
def test_rope_kv_write_from_partial_sums(n_q, n_kv, hd, slices):
    """The q/k/v projection as float slices of K: added in order, rotated, rounded once, written to the packed
    row and to the cache; a row with a negative position is left alone."""
    g = torch.Generator().manual_seed(hd + slices)
    T, page = 40, 64
    width = (n_q + 2 * n_kv) * hd
    parts = torch.randn(slices, T, width, generator=g)
    positions = torch.randint(0, 500, (T,), generator=g).int()
    positions[7] = -1
    theta = 1000.0
    inv = torch.tensor(theta, dtype=torch.float64) ** (-2.0 * torch.arange(hd // 2, dtype=torch.float64) / hd)
    ang = torch.arange(500, dtype=torch.float64)[:, None] * inv[None]
    table = torch.stack([ang.cos(), ang.sin()], -1).float()
    rows = torch.randperm(T * 2, generator=g)[:T].int()          # a place of its own for every token
    rows[11] = -1                                                 # a token the ring does not keep
    kp = torch.zeros(3, n_kv, page, hd, dtype=torch.bfloat16, device=DEV)
    vp = torch.zeros_like(kp)
    out = torch.full((T, width), 7.0, dtype=torch.bfloat16, device=DEV)
    kernels.rope_kv_write_parts(parts.to(DEV), out, positions.to(DEV), table.to(DEV), n_q, n_kv, hd, kp, vp,
                                rows.to(DEV), page)
    total = parts.double().sum(0)
    live = positions >= 0
    pos = positions.clamp(min=0)
    q_ref = plain.rope(total[:, :n_q * hd], pos, hd, theta)
    k_ref = plain.rope(total[:, n_q * hd:(n_q + n_kv) * hd], pos, hd, theta)
    ref = torch.cat([q_ref, k_ref, total[:, (n_q + n_kv) * hd:]], dim=1)
    close(out[live], ref[live], torch.bfloat16)
    assert float((out[7].float() - 7.0).abs().max()) == 0.0
    out, kp, vp = out.cpu(), kp.cpu(), vp.cpu()
    for t in range(T):
        if not live[t] or rows[t] < 0:
            continue
        pg, place = int(rows[t]) // page, int(rows[t]) % page
        assert torch.equal(kp[pg, :, place, :].reshape(-1), out[t, n_q * hd:(n_q + n_kv) * hd])
        assert torch.equal(vp[pg, :, place, :].reshape(-1), out[t, (n_q + n_kv) * hd:])
    written = (kp.float().abs().sum(-1) > 0).sum()
    assert int(written) == n_kv * int((live & (rows >= 0)).sum())   # nothing else was touched


def test_rope_skips_padding_rows():
    qkv = torch.randn(4, 4 * 16).to(DEV)
    before = qkv.clone()
    table = torch.zeros(8, 8, 2)
    table[..., 1] = 1.0   # a quarter turn everywhere
    pos = torch.tensor([-1, 2, -1, 3], dtype=torch.int32, device=DEV)
    kernels.rope_kv_write(qkv, pos, table.to(DEV), 2, 1, 16, 16)
    assert torch.equal(qkv[0], before[0]) and torch.equal(qkv[2], before[2])
    assert not torch.equal(qkv[1, :48], before[1, :48])


# ---------------------------------------------------------------------------
# attention
# ---------------------------------------------------------------------------
def _attention_oracle(q, k, v, n_q, n_kv, hd, scale, cap, window):
    return plain.attention(q, k, v, n_q, n_kv, hd, scale, cap, window)


@pytest.mark.parametrize("dtype,kernel", [(torch.float32, "simt"), (torch.bfloat16, "simt"), (torch.bfloat16, "mma"),
                                          (torch.bfloat16, "tc")])
@pytest.mark.parametrize("n_q,n_kv,hd,window,cap", [(4, 2, 16, 8, 50.0), (6, 1, 32, 16, 20.0), (3, 3, 48, 0, 0.0),
                                                    (8, 4, 256, 100, 50.0), (5, 5, 128, 0, 30.0), (8, 1, 64, 33, 0.0),
                                                    (16, 1, 80, 70, 10.0), (4, 2, 64, 0, 50.0), (32, 16, 128, 0, 50.0),
                                                    (8, 8, 256, 0, 0.0)])
def test_attention_packed(dtype, kernel, n_q, n_kv, hd, window, cap):
    if kernel == "tc" and not kernels.attention_prefill_tc_ok(hd, n_q // n_kv):
        pytest.skip("sizes the tcgen05 kernel leaves to the mma.sync kernel")
    g = torch.Generator().manual_seed(hd + n_q)
    lengths = [1, 37, 150, 64, 300]
    T = sum(lengths)
    width = (n_q + 2 * n_kv) * hd
    qkv = (torch.randn(T, width, generator=g)).to(dtype)
    scale = 0.7 / math.sqrt(hd)
    dq = qkv.to(DEV)
    out = torch.empty(T, n_q * hd, dtype=dtype, device=DEV)
    cu = torch.tensor([0] + list(torch.tensor(lengths).cumsum(0)), dtype=torch.int32, device=DEV)
    kw = dict(n_kv=n_kv, group=n_q // n_kv, head_dim=hd, scale=scale, cap=cap, window=window,
              batch=len(lengths), max_q_len=max(lengths))
    kk, vv = dq[:, n_q * hd:(n_q + n_kv) * hd], dq[:, (n_q + n_kv) * hd:]
    if kernel == "mma":
        kernels.attention_prefill_mma(dq[:, :n_q * hd], out, cu, kk, vv, **kw)
    elif kernel == "tc":
        kernels.attention_prefill_tc(dq[:, :n_q * hd], out, cu, kk, vv, **kw)
        assert kernels.attention_tc_status() == 0
    else:
        kernels.attention_simt(dq[:, :n_q * hd], out, cu, torch.tensor(lengths, dtype=torch.int32, device=DEV),
                               k=kk, v=vv, **kw)
    t = 0
    for n in lengths:
        s = qkv[t:t + n]
        ref = _attention_oracle(s[:, :n_q * hd], s[:, n_q * hd:(n_q + n_kv) * hd], s[:, (n_q + n_kv) * hd:],
                                n_q, n_kv, hd, scale, cap, window)
        close(out[t:t + n], ref, dtype, scale=float(ref.abs().max()))
        t += n


@pytest.mark.parametrize("hd,n_q,n_kv", [(64, 4, 2), (128, 16, 4), (256, 16, 1)])
@pytest.mark.parametrize("first", [1, 63, 64, 65, 127, 128, 129, 300])
def test_attention_tc_keeps_broken_values_of_the_next_sequence_out(hd, n_q, n_kv, first):
    """The last key tile of a sequence holds rows of the next one; their infinities and NaNs stay there."""
    g = torch.Generator().manual_seed(first + hd)
    qkv = torch.randn(first + 90, (n_q + 2 * n_kv) * hd, generator=g).to(torch.bfloat16).to(DEV)
    args = dict(n_kv=n_kv, group=n_q // n_kv, head_dim=hd, scale=hd ** -0.5, cap=30.0, window=0)
    k_at, v_at = n_q * hd, (n_q + n_kv) * hd

    def run(rows, lengths):
        out = torch.empty(rows.shape[0], n_q * hd, dtype=torch.bfloat16, device=DEV)
        cu = torch.tensor([0] + list(torch.tensor(lengths).cumsum(0)), dtype=torch.int32, device=DEV)
        kernels.attention_prefill_tc(rows[:, :k_at], out, cu, rows[:, k_at:v_at], rows[:, v_at:], batch=len(lengths),
                                     max_q_len=max(lengths), n_split=0, **args)
        assert kernels.attention_tc_status() == 0
        return out

    alone = run(qkv[:first].contiguous(), [first])
    qkv[first::2, v_at:] = float("nan")
    qkv[first + 1::2, v_at:] = float("inf")
    assert torch.equal(run(qkv, [first, 90])[:first], alone)


@pytest.mark.parametrize("hd,n_q,n_kv", [(64, 4, 2), (128, 16, 4), (256, 16, 1)])
@pytest.mark.parametrize("cap,gain", [(0.0, 0.3), (30.0, 1.0), (30.0, 3.0), (50.0, 5.0)])
def test_attention_tc_tight_is_as_precise_as_mma(hd, n_q, n_kv, cap, gain):
    """Scores of deviation ``gain``, from flat to a few leading keys: the error against 64 bits of the whole result, over
    some 10^6 entries, is that of the mma.sync kernel (whose tiles are half as wide) but for one part in a hundred."""
    g = torch.Generator().manual_seed(hd + int(10 * gain))
    lengths = [900, 389, 64]
    T = sum(lengths)
    qkv = torch.randn(T, (n_q + 2 * n_kv) * hd, generator=g).to(torch.bfloat16)
    dq = qkv.to(DEV)
    cu = torch.tensor([0] + list(torch.tensor(lengths).cumsum(0)), dtype=torch.int32, device=DEV)
    k_at, v_at = n_q * hd, (n_q + n_kv) * hd
    kw = dict(n_kv=n_kv, group=n_q // n_kv, head_dim=hd, scale=gain * hd ** -0.5, cap=cap, window=0, batch=len(lengths),
              max_q_len=max(lengths))
    ref = torch.empty(T, k_at, dtype=torch.float64, device=DEV)
    for b, n in enumerate(lengths):
        at = sum(lengths[:b])
        rows = dq[at:at + n].double()
        heads = lambda part, count: part.view(n, count, hd).transpose(0, 1)
        q, k, v = heads(rows[:, :k_at], n_q), heads(rows[:, k_at:v_at], n_kv), heads(rows[:, v_at:], n_kv)
        k, v = (t.repeat_interleave(n_q // n_kv, 0) for t in (k, v))
        s = q @ k.transpose(1, 2) * kw["scale"]
        s = cap * torch.tanh(s / cap) if cap else s
        s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device=DEV).triu(1), -torch.inf)
        ref[at:at + n] = (torch.softmax(s, -1) @ v).transpose(0, 1).reshape(n, k_at)

    def error(kernel, **more):
        out = torch.empty(T, k_at, dtype=torch.bfloat16, device=DEV)
        kernel(dq[:, :k_at], out, cu, dq[:, k_at:v_at], dq[:, v_at:], **kw, **more)
        return float((out.double() - ref).norm() / ref.norm())

    mma = error(kernels.attention_prefill_mma)
    for n_split in (0, 5):
        assert error(kernels.attention_prefill_tc, tight=True, n_split=n_split) <= 1.01 * mma
    assert kernels.attention_tc_status() == 0


@pytest.mark.parametrize("n_q,n_kv,hd,window,cap,gain", [(8, 4, 256, 0, 50.0, 40.0), (4, 2, 64, 100, 30.0, 25.0),
                                                         (4, 4, 128, 0, 20.0, 200.0)])
def test_attention_tc_scores_beyond_the_cap(n_q, n_kv, hd, window, cap, gain):
    """Queries scaled so that score * scale / cap runs from near 0 to far beyond 1, where tanh is flat and
    the row's reference maximum sits at the cap: tiles with small scores and tiles with saturated ones
    follow one another within a sequence."""
    g = torch.Generator().manual_seed(5)
    lengths = [300, 700, 129]
    T = sum(lengths)
    qkv = torch.randn(T, (n_q + 2 * n_kv) * hd, generator=g)
    # rows 0-255 of each sequence keep small scores; later query rows are large
    t = 0
    for n in lengths:
        qkv[t + 256:t + n, :n_q * hd] *= gain
        t += n
    qkv = qkv.to(torch.bfloat16)
    scale = 1.0 / math.sqrt(hd)
    dq = qkv.to(DEV)
    out = torch.empty(T, n_q * hd, dtype=torch.bfloat16, device=DEV)
    cu = torch.tensor([0] + list(torch.tensor(lengths).cumsum(0)), dtype=torch.int32, device=DEV)
    kernels.attention_prefill_tc(dq[:, :n_q * hd], out, cu, dq[:, n_q * hd:(n_q + n_kv) * hd], dq[:, (n_q + n_kv) * hd:],
                                 n_kv=n_kv, group=n_q // n_kv, head_dim=hd, scale=scale, cap=cap, window=window,
                                 batch=len(lengths), max_q_len=max(lengths))
    assert kernels.attention_tc_status() == 0
    t = 0
    for n in lengths:
        s = qkv[t:t + n]
        ref = _attention_oracle(s[:, :n_q * hd], s[:, n_q * hd:(n_q + n_kv) * hd], s[:, (n_q + n_kv) * hd:],
                                n_q, n_kv, hd, scale, cap, window)
        close(out[t:t + n], ref, torch.bfloat16, scale=float(ref.abs().max()))
        t += n


@pytest.mark.parametrize("n_q,n_kv,hd,window,cap,lengths", [(8, 4, 256, 512, 50.0, [1500, 130]),
                                                            (8, 4, 256, 0, 50.0, [2100]),
                                                            (4, 2, 128, 0, 30.0, [2100, 700])])
def test_attention_tc_long_prompts(n_q, n_kv, hd, window, cap, lengths):
    """Prompts of many key tiles: 1,500 tokens with a window of 512 (row blocks whose first key tile is
    not tile 0, windows that cut tiles at both ends) and 2,100 tokens without a window."""
    g = torch.Generator().manual_seed(11)
    T = sum(lengths)
    qkv = torch.randn(T, (n_q + 2 * n_kv) * hd, generator=g).to(torch.bfloat16)
    scale = 1.0 / math.sqrt(hd)
    dq = qkv.to(DEV)
    out = torch.empty(T, n_q * hd, dtype=torch.bfloat16, device=DEV)
    cu = torch.tensor([0] + list(torch.tensor(lengths).cumsum(0)), dtype=torch.int32, device=DEV)
    kernels.attention_prefill_tc(dq[:, :n_q * hd], out, cu, dq[:, n_q * hd:(n_q + n_kv) * hd], dq[:, (n_q + n_kv) * hd:],
                                 n_kv=n_kv, group=n_q // n_kv, head_dim=hd, scale=scale, cap=cap, window=window,
                                 batch=len(lengths), max_q_len=max(lengths))
    assert kernels.attention_tc_status() == 0
    t = 0
    for n in lengths:
        s = qkv[t:t + n]
        ref = _attention_oracle(s[:, :n_q * hd], s[:, n_q * hd:(n_q + n_kv) * hd], s[:, (n_q + n_kv) * hd:],
                                n_q, n_kv, hd, scale, cap, window)
        close(out[t:t + n], ref, torch.bfloat16, scale=float(ref.abs().max()))
        t += n


@pytest.mark.parametrize("n_q,n_kv,hd,window,cap,lengths,n_split", [
    (8, 4, 256, 0, 50.0, [2048], None),            # the launcher's own choice (it cuts: 128 blocks on 148 SMs)
    (8, 4, 256, 0, 50.0, [1100], 9),               # every row block in two
    (8, 4, 256, 0, 50.0, [1100], 3),               # only the three heaviest
    (8, 4, 256, 300, 50.0, [1500], 24),            # a window: the first half of a row block ends before some rows' windows begin
    (4, 2, 128, 0, 30.0, [700, 64, 1, 130, 333], 6),   # sequences too short for the cut ranks, and ranks with one tile
    (4, 4, 64, 0, 0.0, [515, 900], 8),
    (2, 1, 256, 128, 50.0, [640], 5)])
def test_attention_tc_row_blocks_cut_in_two_along_the_keys(n_q, n_kv, hd, window, cap, lengths, n_split):
    """The heaviest row blocks as two halves of their keys, merged by the half that finishes second.  One far
    key per sequence (key 3, in the first half of every later row block) is made to carry almost all the
    weight of the last rows, so a lost or mis-scaled first half shows; twice over, so the tickets must have
    gone back to zero."""
    g = torch.Generator().manual_seed(17 + hd)
    T = sum(lengths)
    group = n_q // n_kv
    qkv = torch.randn(T, (n_q + 2 * n_kv) * hd, generator=g)
    t = 0
    for n in lengths:
        if n > 200 and (window == 0 or window > n):
            key = qkv[t + 3, n_q * hd:n_q * hd + hd]
            qkv[t + n - 40:t + n, :hd] = key * 0.5           # head 0 of the last rows looks at key 3
        t += n
    qkv = qkv.to(torch.bfloat16)
    scale = 1.0 / math.sqrt(hd)
    dq = qkv.to(DEV)
    cu = torch.tensor([0] + list(torch.tensor(lengths).cumsum(0)), dtype=torch.int32, device=DEV)
    kw = dict(n_kv=n_kv, group=group, head_dim=hd, scale=scale, cap=cap, window=window, batch=len(lengths),
              max_q_len=max(lengths))
    if n_split is None:
        assert kernels.attention_prefill_tc_split(max(lengths), n_kv, group, window, len(lengths)) > 0
    whole = torch.empty(T, n_q * hd, dtype=torch.bfloat16, device=DEV)
    kernels.attention_prefill_tc(dq[:, :n_q * hd], whole, cu, dq[:, n_q * hd:(n_q + n_kv) * hd], dq[:, (n_q + n_kv) * hd:],
                                 n_split=0, **kw)
    for _ in range(2):
        out = torch.full((T, n_q * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
        kernels.attention_prefill_tc(dq[:, :n_q * hd], out, cu, dq[:, n_q * hd:(n_q + n_kv) * hd], dq[:, (n_q + n_kv) * hd:],
                                     n_split=n_split, **kw)
        assert kernels.attention_tc_status() == 0
        t = 0
        for n in lengths:
            s_ = qkv[t:t + n]
            ref = _attention_oracle(s_[:, :n_q * hd], s_[:, n_q * hd:(n_q + n_kv) * hd], s_[:, (n_q + n_kv) * hd:],
                                    n_q, n_kv, hd, scale, cap, window)
            close(out[t:t + n], ref, torch.bfloat16, scale=float(ref.abs().max()))
            t += n
        # and close to the uncut kernel's result (the same products, another order of two sums)
        assert float((out.float() - whole.float()).abs().max()) <= 2e-2 * float(whole.float().abs().max())


def _paged_case(dtype, n_q, n_kv, hd, window, cap, lengths, page=64, special=None, seed=0, kernel="simt", splits=1):
    """Decode pass: one query per sequence over a scattered, possibly ring-shaped cache."""
    g = torch.Generator().manual_seed(seed)
    B = len(lengths)
    ring = ((window + page - 1) // page * page) if window else (1 << 30)
    scale = 1.0 / math.sqrt(hd)
    ks = [torch.randn(n, n_kv * hd, generator=g).to(dtype) for n in lengths]
    vs = [torch.randn(n, n_kv * hd, generator=g).to(dtype) for n in lengths]
    qs = [torch.randn(1, n_q * hd, generator=g).to(dtype) for _ in lengths]
    if special is not None:
        special(qs, ks, vs)
    pages_per = [min((n + page - 1) // page, ring // page) for n in lengths]
    n_pages = sum(pages_per) + 2
    perm = iter(torch.randperm(n_pages, generator=g).tolist())
    pt = torch.zeros(B, max(pages_per), dtype=torch.int32)
    kp = torch.full((n_pages, n_kv, page, hd), float("nan")).to(dtype)   # what is never written must never be read
    vp = kp.clone()
    for b, n in enumerate(lengths):
        for j in range(pages_per[b]):
            pt[b, j] = next(perm)
        for p in range(max(0, n - ring), n):
            ridx = p % ring
            kp[int(pt[b, ridx // page]), :, ridx % page, :] = ks[b][p].view(n_kv, hd)
            vp[int(pt[b, ridx // page]), :, ridx % page, :] = vs[b][p].view(n_kv, hd)
    q = torch.cat(qs).to(DEV)
    out = torch.empty(B, n_q * hd, dtype=dtype, device=DEV)
    cu = torch.arange(B + 1, dtype=torch.int32, device=DEV)
    kvl = torch.tensor(lengths, dtype=torch.int32, device=DEV)
    kw = dict(n_kv=n_kv, group=n_q // n_kv, head_dim=hd, scale=scale, cap=cap, window=window, batch=B)
    if kernel == "mma":
        kernels.attention_decode_mma(q, out, cu, kvl, kp.to(DEV), vp.to(DEV), pt.to(DEV), ring=ring, page_size=page,
                                     n_splits=splits, **kw)
    else:
        kernels.attention_simt(q, out, cu, kvl, max_q_len=1, k_pages=kp.to(DEV), v_pages=vp.to(DEV),
                               page_table=pt.to(DEV), ring=ring, page_size=page, **kw)
    assert bool(torch.isfinite(out.float()).all()), "a place of the cache that was never written was read"
    for b, n in enumerate(lengths):
        if n > 1200:
            # too long for a matrix per head: the oracle's form for one query (the plain tests tie it to the other)
            ref = plain.attention_last_query(qs[b][0], ks[b], vs[b], n_q, n_kv, hd, scale, cap, window)
        else:
            # oracle over the whole sequence with the query as the last row
            qfull = torch.zeros(n, n_q * hd).to(dtype)
            qfull[-1] = qs[b][0]
            ref = _attention_oracle(qfull, ks[b], vs[b], n_q, n_kv, hd, scale, cap, window)[-1]
        close(out[b], ref, dtype, scale=float(ref.abs().max()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n_q,n_kv,hd,window,cap", [(4, 2, 16, 8, 50.0), (6, 1, 32, 100, 20.0), (3, 3, 48, 0, 0.0),
                                                    (8, 4, 256, 0, 50.0), (8, 4, 256, 70, 50.0)])
def test_attention_paged(dtype, n_q, n_kv, hd, window, cap):
    _paged_case(dtype, n_q, n_kv, hd, window, cap, lengths=[1, 63, 64, 65, 129, 300], seed=hd + window)


@pytest.mark.parametrize("splits", [1, 2, 5, 16])
@pytest.mark.parametrize("n_q,n_kv,hd,window,cap", [(4, 2, 16, 8, 50.0), (6, 1, 32, 100, 20.0), (3, 3, 48, 0, 0.0),
                                                    (8, 4, 256, 0, 50.0), (8, 4, 256, 70, 50.0), (16, 1, 128, 0, 0.0),
                                                    (5, 1, 80, 200, 30.0)])
def test_attention_decode_tensor_cores(splits, n_q, n_kv, hd, window, cap):
    _paged_case(torch.bfloat16, n_q, n_kv, hd, window, cap, lengths=[1, 63, 64, 65, 129, 300, 1000],
                seed=hd + window, kernel="mma", splits=splits)


@pytest.mark.parametrize("splits", [17, 33, 40])
@pytest.mark.parametrize("n_q,n_kv,hd,window,cap", [(8, 4, 256, 0, 50.0), (8, 4, 256, 4096, 50.0), (32, 16, 128, 0, 50.0),
                                                    (6, 1, 32, 0, 20.0)])
def test_attention_decode_many_splits(splits, n_q, n_kv, hd, window, cap):
    """More splits than a warp has lanes (the merge then takes two rounds per thread), as one sequence of
    8,192 keys on four kv heads gets them (37 on 148 SMs); sequences of a few keys beside long ones leave
    most splits empty; with the real window the ring of 64 pages is read through 65 tiles."""
    _paged_case(torch.bfloat16, n_q, n_kv, hd, window, cap, lengths=[5300, 70, 2600, 4161], seed=hd + splits,
                kernel="mma", splits=splits)


def test_attention_decode_far_key_at_the_splits_of_one_long_sequence():
    """One sequence of 8,192 keys: the launch policy gives it 37 splits.  Key 17 carries all the weight."""
    n_q, n_kv, hd = 8, 4, 64
    splits = kernels.decode_splits(1, n_kv, 8192, 0, sms=148)
    assert splits == 37

    def special(qs, ks, vs):
        ks[0][17] = 0
        qs[0][:] = 0
        for g in range(n_kv):
            ks[0][17, g * hd] = 8.0
        for h in range(n_q):
            qs[0][0, h * hd] = 8.0
        vs[0][17] = 5.0

    _paged_case(torch.bfloat16, n_q, n_kv, hd, 0, 0.0, lengths=[8192], special=special, seed=3, kernel="mma",
                splits=splits)


def test_attention_decode_tensor_cores_skips_padding_rows():
    """A row with kv_len 0 is padding: its output is zero and the cache is not read for it."""
    n_q, n_kv, hd = 4, 2, 64
    kp = torch.randn(3, n_kv, 64, hd).to(torch.bfloat16).to(DEV)
    q = torch.randn(3, n_q * hd).to(torch.bfloat16).to(DEV)
    out = torch.full((3, n_q * hd), 7.0, dtype=torch.bfloat16, device=DEV)
    pt = torch.tensor([[0, 1], [0, 0], [2, 0]], dtype=torch.int32, device=DEV)
    for splits in (1, 3):
        kernels.attention_decode_mma(q, out, torch.arange(4, dtype=torch.int32, device=DEV),
                                     torch.tensor([100, 0, 5], dtype=torch.int32, device=DEV), kp, kp, pt,
                                     ring=1 << 30, page_size=64, n_kv=n_kv, group=2, head_dim=hd, scale=0.1, cap=0.0,
                                     window=0, batch=3, n_splits=splits)
        assert float(out[1].float().abs().max()) == 0.0 and float(out[0].float().abs().max()) > 0


@pytest.mark.parametrize("dtype,kernel,splits", [(torch.float32, "simt", 1), (torch.bfloat16, "mma", 1),
                                                 (torch.bfloat16, "mma", 4)])
def test_attention_far_key_stands_out(dtype, kernel, splits):
    """One key hundreds of places back carries almost all the weight: a kernel
    that drops or misplaces a far page cannot pass."""
    n_q, n_kv, hd = 4, 2, 32
    far = 17

    def special(qs, ks, vs):
        for b in range(len(qs)):
            if ks[b].shape[0] <= far:
                continue
            ks[b][far] = 0
            qs[b][:] = 0
            for g in range(n_kv):
                ks[b][far, g * hd] = 8.0
            for h in range(n_q):
                qs[b][0, h * hd] = 8.0
            vs[b][far] = 5.0

    _paged_case(dtype, n_q, n_kv, hd, 0, 0.0, lengths=[400, 700, 18], special=special, seed=3, kernel=kernel,
                splits=splits)


@pytest.mark.parametrize("dtype,kernel,splits", [(torch.float32, "simt", 1), (torch.bfloat16, "mma", 1),
                                                 (torch.bfloat16, "mma", 3)])
def test_attention_window_edge(dtype, kernel, splits):
    """The key exactly `window` places back must be invisible, the one after it visible."""
    n_q, n_kv, hd, window = 2, 1, 16, 70

    def special(qs, ks, vs):
        for b in range(len(qs)):
            n = ks[b].shape[0]
            if n <= window:
                continue
            qs[b][:] = 0
            qs[b][0, 0] = 8.0
            qs[b][0, hd] = 8.0
            ks[b][n - 1 - window] = 0
            ks[b][n - 1 - window, 0] = 40.0      # just outside: would take all the weight if seen
            vs[b][n - 1 - window] = 1000.0
            ks[b][n - window] = 0
            ks[b][n - window, 0] = 6.0           # just inside
            vs[b][n - window] = 3.0

    _paged_case(dtype, n_q, n_kv, hd, window, 0.0, lengths=[71, 128, 129, 500], special=special, seed=4,
                kernel=kernel, splits=splits)


def test_attention_prompt_and_decode_agree_bitwise():
    """The float path gives the same bits for a query whether it runs in a prompt or as a decode step."""
    n_q, n_kv, hd, window, page = 4, 2, 32, 40, 64
    g = torch.Generator().manual_seed(9)
    n = 150
    qkv = torch.randn(n, (n_q + 2 * n_kv) * hd, generator=g).to(DEV)
    out = torch.empty(n, n_q * hd, device=DEV)
    cu = torch.tensor([0, n], dtype=torch.int32, device=DEV)
    kw = dict(n_kv=n_kv, group=2, head_dim=hd, scale=0.2, cap=30.0, window=window)
    kernels.attention_simt(qkv[:, :n_q * hd], out, cu, torch.tensor([n], dtype=torch.int32, device=DEV), batch=1,
                           max_q_len=n, k=qkv[:, n_q * hd:(n_q + n_kv) * hd], v=qkv[:, (n_q + n_kv) * hd:], **kw)
    ring = 64
    kp = torch.zeros(1, n_kv, page, hd, device=DEV)
    vp = torch.zeros_like(kp)
    for p in range(n - ring, n):
        kp[0, :, p % ring, :] = qkv[p, n_q * hd:(n_q + n_kv) * hd].view(n_kv, hd)
        vp[0, :, p % ring, :] = qkv[p, (n_q + n_kv) * hd:].view(n_kv, hd)
    one = torch.empty(1, n_q * hd, device=DEV)
    kernels.attention_simt(qkv[n - 1:n, :n_q * hd].contiguous(), one, torch.tensor([0, 1], dtype=torch.int32, device=DEV),
                           torch.tensor([n], dtype=torch.int32, device=DEV), batch=1, max_q_len=1, k_pages=kp,
                           v_pages=vp, page_table=torch.zeros(1, 1, dtype=torch.int32, device=DEV), ring=ring,
                           page_size=page, **kw)
    assert torch.equal(one[0], out[n - 1])


@pytest.mark.parametrize("options", ["plain", "window", "chunk", "scores"])
@pytest.mark.parametrize("n,n_q,n_kv,hd,vd", [(1, 2, 1, 8, 8), (127, 4, 2, 64, 64), (129, 8, 4, 256, 256), (300, 6, 2, 40, 72),
                                              (260, 16, 1, 128, 200), (385, 3, 3, 256, 128)])
def test_float_attention_gives_the_same_bits_however_it_is_cut(monkeypatch, options, n, n_q, n_kv, hd, vd):
    """Spans of 128 keys walked by one block and shared by several, tiles of 8 and 32 rows, packed keys and pages; against
    the kernel for any sizes, which rows off the 16-byte boundaries go to."""
    g = torch.Generator(device=DEV).manual_seed(n + hd)
    q, k, v = (torch.randn(n, w, generator=g, device=DEV) for w in (n_q * hd, n_kv * hd, n_kv * vd))
    extra = dict(window=0)
    if options == "window":
        extra = dict(window=70)
    if options == "chunk":
        extra = dict(window=0, chunk=100)
    if options == "scores":
        extra = dict(window=0, sink=torch.randn(n_q, generator=g, device=DEV), slopes=torch.rand(n_q, generator=g, device=DEV) / 8,
                     dist_bias=torch.randn(n_q, 50, generator=g, device=DEV))
    cu = torch.tensor([0, n], dtype=torch.int32, device=DEV)
    length = torch.tensor([n], dtype=torch.int32, device=DEV)
    kw = dict(n_kv=n_kv, group=n_q // n_kv, head_dim=hd, v_dim=vd, scale=1.5 / math.sqrt(hd), cap=20.0, batch=1, **extra)
    shared, walked, other = (torch.full((n, n_q * vd), float("nan"), device=DEV) for _ in range(3))
    kernels.attention_simt(q, shared, cu, length, k=k, v=v, max_q_len=n, **kw)
    cut = kernels.attn_f32_splits(1, n_kv, n_q // n_kv, vd, n, n, n, extra["window"], extra.get("chunk", 0))
    assert (cut > 1) == (n > 128)
    off = torch.empty(n, n_q * hd + 1, device=DEV)
    off[:, 1:] = q
    kernels.attention_simt(off[:, 1:], other, cu, length, k=k, v=v, max_q_len=n, **kw)
    close(shared, other.double().cpu(), torch.float32, scale=float(other.abs().max()))
    monkeypatch.setattr(kernels, "attn_f32_splits", lambda *a, **b: 0)
    kernels.attention_simt(q, walked, cu, length, k=k, v=v, max_q_len=n, **kw)
    assert torch.equal(shared, walked)
    # the last query as a decode step over pages in another order, walked and shared
    pages = -(-n // 64)
    order = torch.randperm(pages, generator=g, device=DEV)
    kp, vp = (torch.full((pages, n_kv, 64, w), float("nan"), device=DEV) for w in (hd, vd))
    for p in range(n):
        kp[order[p // 64], :, p % 64], vp[order[p // 64], :, p % 64] = k[p].view(n_kv, hd), v[p].view(n_kv, vd)
    table = order.to(torch.int32).view(1, -1)
    for splits in (0, pages):
        monkeypatch.setattr(kernels, "attn_f32_splits", lambda *a, **b: splits)
        one = torch.full((1, n_q * vd), float("nan"), device=DEV)
        kernels.attention_simt(q[n - 1:], one, torch.tensor([0, 1], dtype=torch.int32, device=DEV), length, k_pages=kp, v_pages=vp,
                               page_table=table, ring=1 << 30, page_size=64, max_q_len=1, **kw)
        assert torch.equal(one[0], shared[n - 1])


@pytest.mark.parametrize("n_q,n_kv,hd,vd", [(8, 1, 256, 256), (8, 1, 8, 8), (5, 1, 40, 24), (6, 2, 136, 200), (16, 4, 64, 16)])
@pytest.mark.parametrize("tokens", [1, 2])
def test_float_attention_of_a_few_rows_gives_the_bits_of_more(monkeypatch, n_q, n_kv, hd, vd, tokens):
    """Up to eight rows in clusters that share a span, value rows of fewer entries than the blocks' shares, several spans and a
    bound that does not hold, against the same rows walked by one block."""
    g = torch.Generator(device=DEV).manual_seed(hd + vd)
    group = n_q // n_kv
    tokens = 1 if tokens * group > 8 else tokens
    lengths = [2, 128, 129, 500, 31]
    B, table = len(lengths), torch.randperm(40, generator=g, device=DEV).to(torch.int32).view(5, 8)
    kp, vp = torch.randn(40, n_kv, 64, hd, generator=g, device=DEV), torch.randn(40, n_kv, 64, vd, generator=g, device=DEV)
    q = torch.randn(B * tokens, n_q * hd, generator=g, device=DEV)
    monkeypatch.setattr(kernels, "attn_f32_worth_sharing", lambda *a, **kw: True)
    outs = []
    for splits in (0, 4, 2):                                 # walked; shared; shared, with spans left for the last share
        monkeypatch.setattr(kernels, "attn_f32_splits", lambda *a, **kw: splits)
        outs.append(torch.full((B * tokens, n_q * vd), float("nan"), device=DEV))
        kernels.attention_simt(q, outs[-1], torch.arange(0, B * tokens + 1, tokens, dtype=torch.int32, device=DEV),
                               torch.tensor(lengths, dtype=torch.int32, device=DEV), n_kv=n_kv, group=group, head_dim=hd, v_dim=vd,
                               scale=hd ** -0.5, cap=30.0, window=0, batch=B, max_q_len=tokens, k_pages=kp, v_pages=vp,
                               page_table=table, ring=1 << 30, page_size=64)
    assert torch.equal(outs[0], outs[1]) and not bool(outs[0].isnan().any())
    close(outs[2], outs[0].double().cpu(), torch.float32, scale=float(outs[0].abs().max()))      # (a share's spans are merged first)


@pytest.mark.parametrize("n_kv,hd,vd", [(2, 64, 64), (4, 256, 256), (3, 40, 136)])
@pytest.mark.parametrize("batch", [6, 60])
def test_float_attention_of_few_rows_in_clusters_and_a_block_a_span(monkeypatch, batch, n_kv, hd, vd):
    """Four spans of each sequence: in clusters where they are fewer than SMs, else a block each; the bits of one that walks."""
    assert (batch * n_kv * 4 <= kernels.device_sms()) == (batch == 6)
    g = torch.Generator(device=DEV).manual_seed(hd + batch)
    pages = batch * 8
    table = torch.randperm(pages, generator=g, device=DEV).to(torch.int32).view(batch, 8)
    kp, vp = torch.randn(pages, n_kv, 64, hd, generator=g, device=DEV), torch.randn(pages, n_kv, 64, vd, generator=g, device=DEV)
    q = torch.randn(batch, 2 * n_kv * hd, generator=g, device=DEV)
    lengths = torch.randint(1, 513, (batch,), generator=g, device=DEV).to(torch.int32)
    monkeypatch.setattr(kernels, "attn_f32_worth_sharing", lambda *a, **kw: True)
    outs = []
    for splits in (0, 4):
        monkeypatch.setattr(kernels, "attn_f32_splits", lambda *a, **kw: splits)
        outs.append(torch.full((batch, 2 * n_kv * vd), float("nan"), device=DEV))
        kernels.attention_simt(q, outs[-1], torch.arange(batch + 1, dtype=torch.int32, device=DEV), lengths, n_kv=n_kv, group=2,
                               head_dim=hd, v_dim=vd, scale=hd ** -0.5, cap=30.0, window=0, batch=batch, max_q_len=1, k_pages=kp,
                               v_pages=vp, page_table=table, ring=1 << 30, page_size=64)
    assert torch.equal(outs[0], outs[1]) and not bool(outs[0].isnan().any())


@pytest.mark.parametrize("rows", [16, 32])
@pytest.mark.parametrize("hd,vd", [(64, 64), (64, 128), (40, 72), (256, 256), (128, 200)])
@pytest.mark.parametrize("n", [131, 300])
def test_float_attention_of_a_prompt_in_tiles_of_16_and_32_rows(monkeypatch, n, hd, vd, rows):
    """Shared spans in either tile, every number of value columns a thread: the bits of blocks that walk (tiles of 32)."""
    batch, n_kv = (1, 3) if rows == 16 else (3, 12)
    tiles, spans = -(-n * 2 // 32), -(-n // 128)
    assert (2 * tiles * n_kv * batch * (spans + 1) <= 5 * kernels.device_sms()) == (rows == 16)
    g = torch.Generator(device=DEV).manual_seed(n + hd + vd)
    lengths = [n, n - 37, 5][:batch]
    T, n_q = sum(lengths), 2 * n_kv
    q, k, v = (torch.randn(T, w, generator=g, device=DEV) for w in (n_q * hd, n_kv * hd, n_kv * vd))
    cu = torch.tensor([0] + [sum(lengths[:i + 1]) for i in range(batch)], dtype=torch.int32, device=DEV)
    monkeypatch.setattr(kernels, "attn_f32_worth_sharing", lambda *a, **kw: True)
    outs = []
    for cut in (spans, 0):
        monkeypatch.setattr(kernels, "attn_f32_splits", lambda *a, **kw: cut)
        outs.append(torch.full((T, n_q * vd), float("nan"), device=DEV))
        kernels.attention_simt(q, outs[-1], cu, torch.tensor(lengths, dtype=torch.int32, device=DEV), n_kv=n_kv, group=2, head_dim=hd,
                               v_dim=vd, scale=hd ** -0.5, cap=20.0, window=0, batch=batch, max_q_len=n, k=k, v=v)
    assert torch.equal(outs[0], outs[1]) and not bool(outs[0].isnan().any())


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("lengths", [[3], [32, 5, 1], [33, 64, 20], [65, 7, 96], [97, 40], [129, 160, 31]])
@pytest.mark.parametrize("window,chunk", [(0, 0), (1, 0), (40, 0), (70, 0), (0, 33)])
def test_float_attention_of_parts_of_spans(monkeypatch, lengths, window, chunk, shared):
    """One, two and all 32-key parts of a span, at either end of it, with prompts short enough for small stages; a row's bits
    are those of a launch with stages for whole spans, and all is close to 64 bits."""
    g = torch.Generator(device=DEV).manual_seed(sum(lengths) + window)
    n_q, n_kv, hd, vd = 6, 3, 24, 40
    T, B = sum(lengths), len(lengths)
    q, k, v = (torch.randn(T, w, generator=g, device=DEV) for w in (n_q * hd, n_kv * hd, n_kv * vd))
    cu = torch.tensor([0] + list(torch.tensor(lengths).cumsum(0)), dtype=torch.int32, device=DEV)
    length = torch.tensor(lengths, dtype=torch.int32, device=DEV)
    monkeypatch.setattr(kernels, "attn_f32_worth_sharing", lambda *a, **kw: shared)
    kw = dict(n_kv=n_kv, group=2, head_dim=hd, v_dim=vd, scale=hd ** -0.5, cap=20.0, window=window, chunk=chunk, batch=B, k=k, v=v)
    out, wide = (torch.full((T, n_q * vd), float("nan"), device=DEV) for _ in range(2))
    kernels.attention_simt(q, out, cu, length, max_q_len=max(lengths), **kw)
    kernels.attention_simt(q, wide, cu, length, max_q_len=max(max(lengths), 300), **kw)      # stages for whole spans
    assert torch.equal(out, wide)
    for b, n in enumerate(lengths):
        at = int(cu[b])
        heads = lambda t, count: t[at:at + n].double().view(n, count, -1).transpose(0, 1)
        kk, vv = (heads(t, n_kv).repeat_interleave(2, 0) for t in (k, v))
        s = heads(q, n_q) @ kk.transpose(1, 2) * hd ** -0.5
        s = 20.0 * torch.tanh(s / 20.0)
        p, j = torch.arange(n, device=DEV).view(-1, 1), torch.arange(n, device=DEV)
        seen = (j <= p) & ((p - j < window) if window else (j >= 0)) & ((j >= p - p % chunk) if chunk else (j >= 0))
        ref = torch.softmax(s.masked_fill(~seen, -torch.inf), -1) @ vv
        close(out[at:at + n], ref.transpose(0, 1).reshape(n, -1).cpu(), torch.float32, scale=float(ref.abs().max()))


@pytest.mark.parametrize("options", [dict(keep_first=4, chunk=8), dict(keep_first=-1), dict(keep_first=-1, window=5)])
def test_float_attention_refuses_the_options_that_exclude_each_other(options):
    x = torch.zeros(8, 32, device=DEV)
    with pytest.raises(kernels.KernelError):
        kernels.attention_simt(x, torch.empty_like(x), torch.tensor([0, 8], dtype=torch.int32, device=DEV),
                               torch.tensor([8], dtype=torch.int32, device=DEV), k=x, v=x, batch=1, max_q_len=8,
                               **{**dict(n_kv=1, group=1, head_dim=32, scale=1.0, cap=0.0, window=0), **options})


@pytest.mark.parametrize("bound", [700, 512, 100])
def test_float_attention_with_a_bound_on_the_keys(monkeypatch, bound):
    """A bound cuts the work; one that does not hold costs no keys."""
    g = torch.Generator(device=DEV).manual_seed(bound)
    lengths, n_kv, hd = [700, 3, 450, 128], 2, 32
    B = len(lengths)
    table = torch.randperm(64 * B, generator=g, device=DEV).to(torch.int32).view(B, 64)
    kp, vp = (torch.randn(64 * B, n_kv, 64, hd, generator=g, device=DEV) for _ in range(2))
    q = torch.randn(B, n_kv * 2 * hd, generator=g, device=DEV)
    monkeypatch.setattr(kernels, "attn_f32_worth_sharing", lambda *a, **kw: True)
    outs = []
    for keys in (None, bound):
        outs.append(torch.full_like(q, float("nan")))
        kernels.attention_simt(q, outs[-1], torch.arange(B + 1, dtype=torch.int32, device=DEV),
                               torch.tensor(lengths, dtype=torch.int32, device=DEV), n_kv=n_kv, group=2, head_dim=hd, scale=0.2, cap=0.0,
                               window=0, batch=B, max_q_len=1, k_pages=kp, v_pages=vp, page_table=table, ring=1 << 30, page_size=64,
                               max_keys=keys)
    if bound >= max(lengths):
        assert torch.equal(*outs)
    close(outs[1], outs[0].double().cpu(), torch.float32)


@pytest.mark.parametrize("window", [1, 100, 128, 129, 257, 300, 400])
@pytest.mark.parametrize("shared", [False, True])
def test_float_attention_in_wrapped_rings_gives_the_bits_of_the_prompt(monkeypatch, window, shared):
    """Several sequences decoded from rings of their window's pages, up to four spans wide and many times wrapped, against
    the last tokens of the same sequences as packed prompts: the same bits, walked and shared."""
    g = torch.Generator(device=DEV).manual_seed(window)
    n_q, n_kv, hd, vd = 4, 2, 16, 24
    lengths = [1, 130, 700, 641, 385, 512]
    T, B, ring = sum(lengths), len(lengths), -(-window // 64) * 64
    q, k, v = (torch.randn(T, w, generator=g, device=DEV) for w in (n_q * hd, n_kv * hd, n_kv * vd))
    cu = torch.tensor([0] + list(torch.tensor(lengths).cumsum(0)), dtype=torch.int32, device=DEV)
    length = torch.tensor(lengths, dtype=torch.int32, device=DEV)
    monkeypatch.setattr(kernels, "attn_f32_worth_sharing", lambda *a, **kw: shared)
    kw = dict(n_kv=n_kv, group=2, head_dim=hd, v_dim=vd, scale=0.5, cap=0.0, window=window, batch=B)
    packed = torch.full((T, n_q * vd), float("nan"), device=DEV)
    kernels.attention_simt(q, packed, cu, length, max_q_len=max(lengths), k=k, v=v, **kw)
    per = ring // 64
    table = torch.randperm(B * per, generator=g, device=DEV).to(torch.int32).view(B, per)
    kp, vp = torch.zeros(B * per, n_kv, 64, hd, device=DEV), torch.zeros(B * per, n_kv, 64, vd, device=DEV)
    for b, n in enumerate(lengths):
        at = int(cu[b])
        for p in range(max(0, n - ring), n):
            page = int(table[b, p % ring // 64])
            kp[page, :, p % 64], vp[page, :, p % 64] = k[at + p].view(n_kv, hd), v[at + p].view(n_kv, vd)
    ends = (cu[1:] - 1).long()
    one = torch.full((B, n_q * vd), float("nan"), device=DEV)
    kernels.attention_simt(q[ends], one, torch.arange(B + 1, dtype=torch.int32, device=DEV), length, max_q_len=1, k_pages=kp,
                           v_pages=vp, page_table=table, ring=ring, page_size=64, **kw)
    assert torch.equal(one, packed[ends])


@pytest.mark.parametrize("options", ["plain", "sink", "bias", "one row"])
@pytest.mark.parametrize("hd,n_kv,splits", [(256, 4, 2), (144, 2, 4), (64, 4, 3)])
@pytest.mark.parametrize("batch,longest_first", [(98, True), (98, False), (512, True), (513, True)])
def test_decode_attention_gives_the_same_bits_whatever_runs_beside_it(options, hd, n_kv, splits, batch, longest_first):
    """More blocks than two rounds hold (two blocks to an SM with large heads, the longest sequences first) against every
    sequence alone (a block to an SM): unequal and equal lengths, one key, a page's edges, padding rows in between."""
    g = torch.Generator(device=DEV).manual_seed(hd + splits)
    lengths = [0, 1, 64, 65, 700, 128, 0, 129, 63, 64] + [1 + 37 * i % 500 for i in range(batch - 10)]
    B, group, W = len(lengths), 2, 11
    assert splits * n_kv * B > 2 * kernels.device_sms(DEV)
    pages = torch.randn(B * W, n_kv, 64, hd, generator=g, device=DEV).to(torch.bfloat16)
    values = pages if options == "one row" else torch.randn(B * W, n_kv, 64, hd, generator=g, device=DEV).to(torch.bfloat16)
    table = torch.randperm(B * W, generator=g, device=DEV).to(torch.int32).view(B, W)
    q = torch.randn(B, n_kv * group * hd, generator=g, device=DEV).to(torch.bfloat16)
    extra = dict(sink=torch.randn(n_kv * group, generator=g, device=DEV)) if options == "sink" else {}
    if options == "bias":
        extra = dict(dist_bias=torch.randn(n_kv * group, 100, generator=g, device=DEV))
    kw = dict(ring=1 << 30, page_size=64, n_kv=n_kv, group=group, head_dim=hd, scale=hd ** -0.5, cap=20.0, window=300,
              n_splits=splits, **extra)
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)
    out = torch.full_like(q, 7.0)
    kernels.attention_decode_mma(q, out, torch.arange(B + 1, dtype=torch.int32, device=DEV), i32(*lengths), pages, values, table,
                                 batch=B, longest_first=longest_first, **kw)
    for b in range(B) if batch < 100 else range(0, B, 17):
        one = torch.full_like(q[b:b + 1], 7.0)
        kernels.attention_decode_mma(q[b:b + 1], one, i32(0, 1), i32(lengths[b]), pages, values, table[b:b + 1], batch=1, **kw)
        assert torch.equal(out[b], one[0]), (b, lengths[b])


@pytest.mark.parametrize("activation,limit", [("gelu_tanh", 0.0), ("silu", 0.0), ("clamped_gate", 7.0)])
def test_few_tokens_have_the_same_activation_on_both_products(activation, limit):
    """One weight for every output, so that the sums are exact: what is left is the activation, to the last bit."""
    g = torch.Generator(device=DEV).manual_seed(3)
    x = torch.eye(16, 64, device=DEV).to(torch.bfloat16)
    w = (3 * torch.randn(2 * 8192, 64, generator=g, device=DEV)).to(torch.bfloat16)
    few, stream = (torch.empty(16, 8192, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    kernels.skinny_gemm(x, w, few, "gated", activation, limit=limit)
    kernels.gemm_stream(x, w, stream, "gated", activation, limit=limit)
    assert torch.equal(few, stream)


def test_kernels_refuse_what_they_cannot_do():
    q = torch.zeros(2, 2 * 520, device=DEV)
    with pytest.raises(kernels.KernelError):                # a head beyond the exact kernel's 512
        kernels.attention_simt(q, torch.empty_like(q), torch.tensor([0, 2], dtype=torch.int32, device=DEV),
                               torch.tensor([2], dtype=torch.int32, device=DEV), n_kv=1, group=2, head_dim=520,
                               scale=1.0, cap=0.0, window=0, batch=1, max_q_len=2, k=q, v=q)
    with pytest.raises(kernels.KernelError):
        kernels.gated_act(torch.zeros(1, 8, device=DEV), torch.zeros(1, 4, device=DEV), "relu")
    with pytest.raises(kernels.KernelError):
        kernels.embed_scale(torch.zeros(1, dtype=torch.int32), torch.zeros(4, 4), 1.0, torch.zeros(1, 4))


@pytest.mark.parametrize("n_q,n_kv,hd,K,M", [(4, 2, 16, 64, 5), (6, 1, 32, 96, 3), (8, 4, 256, 2304, 8), (3, 1, 48, 72, 16),
                                             (5, 5, 64, 136, 9)])
def test_qkv_product_with_rotation_and_cache_write(n_q, n_kv, hd, K, M):
    """The few-token q/k/v product whose epilogue rotates q and k and writes k, v into the pages:
    against float64, with a padding row (nothing written) and a row that is not kept."""
    from brolm_b200 import kernels
    g = torch.Generator().manual_seed(hd * 7 + K)
    width, page, pages, half = (n_q + 2 * n_kv) * hd, 64, 4, hd // 2
    w = (torch.randn(width, K, generator=g) * 0.1).to(DEV).bfloat16()
    x = torch.randn(M, K, generator=g).to(DEV).bfloat16()
    pos_list = [3, 70, -1, 0, 129] + list(range(5, 16))
    row_list = [3, 64 + 6, 9, -1, 2 * 64 + 1] + list(range(200, 211))
    pos = torch.tensor(pos_list[:M], dtype=torch.int32, device=DEV)
    crow = torch.tensor(row_list[:M], dtype=torch.int32, device=DEV)
    ang = torch.arange(256, dtype=torch.float64)[:, None] * (10000.0 ** (-2.0 * torch.arange(half, dtype=torch.float64) / hd))
    table = torch.stack([ang.cos(), ang.sin()], -1).float().to(DEV).contiguous()
    for use_table, use_pages in ((True, True), (False, True), (True, False)):
        out = torch.full((M, width), 7.0, dtype=torch.bfloat16, device=DEV)
        k_pages = torch.zeros(pages, n_kv, page, hd, dtype=torch.bfloat16, device=DEV)
        v_pages = torch.zeros_like(k_pages)
        kernels.skinny_qkv_rope(x, w, out, pos, table if use_table else None, n_q, n_kv, hd,
                                k_pages if use_pages else None, v_pages if use_pages else None,
                                crow if use_pages else None, page)
        src = (x.double() @ w.double().t()).view(M, n_q + 2 * n_kv, hd)
        want = src.clone()
        if use_table:
            for t in range(M):
                p = pos_list[t]
                if p >= 0:
                    c, s = table[p, :, 0].double(), table[p, :, 1].double()
                    a, b = src[t, :n_q + n_kv, :half], src[t, :n_q + n_kv, half:]
                    want[t, :n_q + n_kv, :half] = a * c - b * s
                    want[t, :n_q + n_kv, half:] = a * s + b * c
        got = out.double().view(M, n_q + 2 * n_kv, hd)
        kept = set()
        for t in range(M):
            if pos_list[t] < 0:
                assert (got[t] == 7.0).all()
                continue
            err = (got[t] - want[t]).abs()
            assert (err <= 2.0 ** -8 * want[t].abs() + 1e-5 * want[t].abs().max()).all()      # one rounding
            r = row_list[t]
            if use_pages and r >= 0:
                kept.add(r)
                assert torch.equal(k_pages[r // page, :, r % page].double(), got[t, n_q:n_q + n_kv])
                assert torch.equal(v_pages[r // page, :, r % page].double(), got[t, n_q + n_kv:])
        mask = torch.ones(pages * page, dtype=torch.bool)
        mask[list(kept)] = False
        for pg in (k_pages, v_pages):
            assert (pg.permute(0, 2, 1, 3).reshape(pages * page, -1)[mask.to(DEV)] == 0).all()
