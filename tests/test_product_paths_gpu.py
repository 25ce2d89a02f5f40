"""b200_gemm on one path at a time, at the sizes where tiles, splits and loads have their edges, in every
operand layout, against an fp64 product of the values the device stores."""
import pytest
import torch

from gpu_util import MODES, TOL

pytestmark = pytest.mark.gpu

# (m, n, k, groups, red): extents at, below and above the tiles (8, 16, 32, 64, 128 columns, 64 and 128 rows,
# k-tiles of 32 floats / 64 halves), the exchanged form (m <= 32 < n), splits over a cluster and over scratch
SIZES = [
    (1, 1, 17, 1, 1), (128, 8, 512, 1, 1), (129, 9, 513, 1, 1), (130, 16, 1000, 2, 1), (10, 300, 77, 1, 1), (33, 31, 4096, 1, 1),
    (256, 256, 256, 1, 1), (64, 64, 64, 3, 1), (65, 63, 33, 3, 1), (200, 136, 264, 1, 3), (515, 387, 201, 2, 1), (384, 320, 2048, 1, 1),
]


def product(a, b, ta, tb, m, n, k):
    """Column-major opA(a) . opB(b) of flat arrays, as a flat array."""
    a = a.view(m, k) if ta else a.view(k, m).T
    b = b.view(k, n).T if tb else b.view(n, k)      # n x k
    return (b @ a.T).reshape(-1)                     # n rows of m: column-major m x n


@pytest.mark.parametrize("path", [2, 4, 5, 6], ids=["tcgen05", "mma_sync", "tcgen05_self_fed", "serial"])
@pytest.mark.parametrize("mode", list(MODES))
@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
def test_paths_at_their_edges(ctx, path, mode, layout):
    if path == 5 and mode in ("tf32", "fp16"):
        pytest.skip("the self-fed kernel is for the fp32 modes")
    if path == 6 and mode == "fp16":
        pytest.skip("the serial kernel is for fp32 storage")
    ta, tb = (int(c == "t") for c in layout)
    kind = torch.float16 if mode == "fp16" else torch.float32
    gen = torch.Generator(device="cuda")
    gen.manual_seed(7)
    for m, n, k, groups, red in SIZES:
        for offset in (0, 1):                        # 1: nothing is aligned
            count = groups * red
            a, b = (torch.randn(count * s + 1, device="cuda", generator=gen).to(kind)[offset:offset + count * s] for s in (m * k, k * n))
            c = torch.randn(groups * m * n + 9, device="cuda", generator=gen).to(kind)[offset:]
            before = c.clone()
            accumulate = (m + n) % 2 == 0
            ctx.gemm(MODES[mode], ta, tb, a.data_ptr(), b.data_ptr(), c.data_ptr(), m, n, k, groups, red,
                     m * k * red if groups > 1 else 0, m * k if red > 1 else 0, k * n * red if groups > 1 else 0,
                     k * n if red > 1 else 0, m * n, accumulate, path)
            assert ctx.status_poll() == 0
            a, b, old = a.double().view(count, -1), b.double().view(count, -1), before.double()
            want = torch.cat([sum(product(a[g * red + r], b[g * red + r], ta, tb, m, n, k) for r in range(red)) for g in range(groups)])
            size = want.norm()                       # errors scale with the product, whatever it is added to
            got = c[:groups * m * n].double() - (old[:groups * m * n] if accumulate else 0)
            # half storage: the sum is rounded once, 2^-11 of its own size
            slack = 2.0 ** -11 * (want + old[:groups * m * n]).norm() if mode == "fp16" and accumulate else 0.0
            if m * n > 1:                            # (a single value may cancel to nothing)
                assert (got - want).norm() <= TOL[mode] * size + slack, (m, n, k, groups, red, offset)
            assert torch.equal(c[groups * m * n:], before[groups * m * n:]), "wrote past the result"


@pytest.mark.parametrize("mode", ["fp16", "tf32", "3xtf32"])
def test_padded_lines_are_shared_inside_one_backward_call(ctx, mode):
    """Operands whose lines TMA cannot address: gy's padded copy serves both gradients of one call (one
    hit), and nothing of it outlives the call."""
    di, dj, dk, n = 515, 389, 131, 6
    kind = torch.float16 if mode == "fp16" else torch.float32
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    a, b, gy = (torch.randn(n * s, device="cuda", generator=gen).to(kind) for s in (di * dj, dj * dk, di * dk))
    ga, gb = torch.empty_like(a), torch.empty_like(b)
    ctx.set_path_policy(2)
    try:
        s0 = ctx.operand_cache_stats()
        ctx.matmul_bw_ex(MODES[mode], a.data_ptr(), b.data_ptr(), gy.data_ptr(), ga.data_ptr(), gb.data_ptr(), di, dj, dk, n, n,
                         False, False)
        s1 = ctx.operand_cache_stats()
    finally:
        ctx.set_path_policy(0)
    assert s1["hits"] - s0["hits"] == 1 and s1["entries"] == 0, (s0, s1)
    a64, b64, gy64 = a.double().view(n, dj, di), b.double().view(n, dk, dj), gy.double().view(n, dk, di)
    want_a = torch.einsum("nki,nkj->nji", gy64, b64)
    want_b = torch.einsum("nji,nki->nkj", a64, gy64)
    for got, want in ((ga, want_a), (gb, want_b)):
        assert (got.double().view_as(want) - want).norm() <= TOL[mode] * want.norm()


@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
def test_sums_of_the_fp32_mode_do_not_depend_on_the_kernel(ctx, layout):
    """Up to 1024 terms are summed in one order: both tcgen05 kernels give the same bits, with tiles of 32, 64
    and 96 columns, with and without slices, at ragged ends of all three extents."""
    ta, tb = (int(c == "t") for c in layout)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(11)
    for m, n, k, groups in ((800, 200, 784, 1), (256, 1024, 256, 1), (129, 33, 1024, 1), (515, 97, 999, 1), (1000, 300, 515, 2), (64, 70, 40, 3)):
        a, b = (torch.randn(groups * s, device="cuda", generator=gen) for s in (m * k, k * n))
        got = []
        for path in (2, 5):
            c = torch.empty(groups * m * n, device="cuda")
            ctx.gemm(MODES["3xtf32"], ta, tb, a.data_ptr(), b.data_ptr(), c.data_ptr(), m, n, k, groups, 1, m * k, 0, k * n, 0, m * n, False, path)
            got.append(c)
        assert ctx.status_poll() == 0
        assert torch.equal(*got), (m, n, k, groups)


@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
def test_tiny_products_carry_infinities_and_nans_as_fp32_does(ctx, layout):
    """An infinite term is an infinite sum (not the nan of inf - inf or inf * 0 inside a split), a nan a nan."""
    ta, tb = (int(c == "t") for c in layout)
    for m, n, k in ((48, 72, 96), (9, 300, 50), (200, 8, 1000)):
        a, b = torch.ones(m * k, device="cuda"), torch.full((k * n,), 0.5, device="cuda")
        at = lambda i, p: i * k + p if ta else p * m + i
        a[at(0, 3)], a[at(1, 5)], a[at(2, 0)] = float("inf"), float("-inf"), float("nan")
        a[at(3, 1)], a[at(3, 2)] = float("inf"), float("-inf")
        a[at(4, 7)] = 3.4e38
        want = product(a, b, ta, tb, m, n, k)
        for mode in ("3xtf32", "tf32", "3xfp16"):
            for path in (0, 4):
                c = torch.empty(m * n, device="cuda")
                ctx.gemm(MODES[mode], ta, tb, a.data_ptr(), b.data_ptr(), c.data_ptr(), m, n, k, 1, 1, 0, 0, 0, 0, 0, False, path)
                assert ctx.status_poll() == 0
                got, fine = c.view(n, m), want.view(n, m)
                assert torch.equal(torch.isnan(got), torch.isnan(fine)), (m, n, k, mode, path)
                finite = torch.isfinite(fine)
                assert torch.equal(got[~finite & ~torch.isnan(fine)], fine[~finite & ~torch.isnan(fine)])
                assert ((got - fine)[finite].abs() <= 1e-5 * fine[finite].abs()).all()


@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
def test_serial_products_have_the_cuda_core_kernels_bits(ctx, layout):
    ta, tb = (int(c == "t") for c in layout)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(12)
    for m, n, k, groups, red in ((10, 200, 800, 1, 1), (1, 1, 17, 1, 1), (8, 16, 128, 1, 1), (9, 17, 129, 3, 1), (33, 31, 127, 1, 5), (7, 300, 257, 2, 1)):
        count = groups * red
        a, b = (torch.randn(count * s, device="cuda", generator=gen) for s in (m * k, k * n))
        c = torch.randn(groups * m * n, device="cuda", generator=gen)
        got = []
        for path in (1, 6):
            out = c.clone()
            ctx.gemm(MODES["3xtf32"], ta, tb, a.data_ptr(), b.data_ptr(), out.data_ptr(), m, n, k, groups, red, m * k if groups > 1 else 0,
                     m * k if red > 1 else 0, k * n if groups > 1 else 0, k * n if red > 1 else 0, m * n, m % 2 == 0, path)
            got.append(out)
        assert ctx.status_poll() == 0
        assert torch.equal(*got), (m, n, k, groups, red)


# nans: what the GPU's own arithmetic makes (0x7fffffff), its negative, ones that a carry or a cut would turn into an infinity
NAN_BITS = (0x7fffffff, -1, 0x7f800001, -0x7fffff, 0x7fc00000)


@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("mode", ["3xtf32", "tf32", "3xfp16"])
def test_no_nan_of_an_operand_is_lost(ctx, mode, layout):
    """Whatever the bits of a nan, the whole row (column) of sums that it is a term of is nan, and nothing else is:
    the split into two terms must keep it in one of them.  Sizes on either side of the tiny ones."""
    ta, tb = (int(c == "t") for c in layout)
    inf = torch.full((1,), float("inf"), device="cuda")
    for m, n, k in ((48, 72, 96), (9, 300, 50), (200, 8, 1000), (256, 256, 320), (300, 96, 1100)):
        for side in (0, 1):
            a, b = torch.ones(m * k, device="cuda"), torch.full((k * n,), 0.5, device="cuda")
            x, lines, by_k = ((a, m, ta), (b, n, not tb))[side]
            at = lambda i, p: i * k + p if by_k else p * lines + i
            for i, bits in enumerate(NAN_BITS):
                x.view(torch.int32)[at(i, 7 * i + 3)] = bits
            x[at(5, 0):at(5, 0) + 1] = inf - inf          # computed on the device
            want = torch.zeros(n, m, dtype=torch.bool, device="cuda")
            (want if side else want.T)[:6] = True
            for path in (0, 4, 5, 6) if mode != "tf32" else (0, 4, 6):
                if mode == "tf32" and n >= 16 and m * n * k >= 2097152:
                    continue                               # (not split: 0x7f800001 cut to TF32 is an infinity)
                c = torch.empty(m * n, device="cuda")
                ctx.gemm(MODES[mode], ta, tb, a.data_ptr(), b.data_ptr(), c.data_ptr(), m, n, k, 1, 1, 0, 0, 0, 0, 0, False, path)
                assert ctx.status_poll() == 0
                assert torch.equal(torch.isnan(c.view(n, m)), want), (m, n, k, side, path)


# two batch axes: every matrix of the batch its own, and the sum over `red` of them
TWO_AXES = [(256, 256, 20, 8, 3), (256, 256, 100, 4, 5), (515, 129, 333, 2, 3), (48, 40, 30, 3, 2), (128, 512, 700, 2, 2)]


def two_axes_error(ctx, mode, layout, size, path):
    """Relative error (norms) of such a product against 64 bits."""
    ta, tb = (int(c == "t") for c in layout)
    m, n, k, groups, red = size
    kind = torch.float16 if mode == "fp16" else torch.float32
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    a, b = (torch.rand(groups * red * s, device="cuda", generator=gen).sub_(0.5).to(kind) for s in (m * k, k * n))
    c = torch.empty(groups * m * n, device="cuda", dtype=kind)
    ctx.gemm(MODES[mode], ta, tb, a.data_ptr(), b.data_ptr(), c.data_ptr(), m, n, k, groups, red, m * k * red, m * k,
             k * n * red, k * n, m * n, False, path)
    assert ctx.status_poll() == 0
    a, b = a.double().view(groups * red, -1), b.double().view(groups * red, -1)
    want = torch.cat([sum(product(a[g * red + r], b[g * red + r], ta, tb, m, n, k) for r in range(red)) for g in range(groups)])
    return float((c.double() - want).norm() / want.norm())


@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("mode", list(MODES))
def test_two_batch_axes_are_taken_in_every_mode(ctx, mode, layout):
    """No kernel of planes takes them, so the choice has to end at one that does, whatever the length of the sum."""
    for size in TWO_AXES:
        assert two_axes_error(ctx, mode, layout, size, 0) <= TOL[mode], size


@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("mode", ["3xtf32", "tf32", "3xfp16"])
def test_two_batch_axes_keep_fp32_sums(ctx, mode, layout):
    """As precise as the CUDA cores (path 1), the single-pass mode included, and infinite where those are."""
    for size in TWO_AXES:
        assert two_axes_error(ctx, mode, layout, size, 0) <= 1.05 * two_axes_error(ctx, mode, layout, size, 1), size
    ta, tb = (int(c == "t") for c in layout)
    m, n, k, groups, red = 256, 256, 100, 2, 3
    a, b = torch.ones(groups * red * m * k, device="cuda"), torch.full((groups * red * k * n,), 0.5, device="cuda")
    at = (red + 1) * m * k                                # second matrix of the second group, element (0, 0)
    a[at] = float("inf")
    c = torch.empty(groups * m * n, device="cuda")
    ctx.gemm(MODES[mode], ta, tb, a.data_ptr(), b.data_ptr(), c.data_ptr(), m, n, k, groups, red, m * k * red, m * k, k * n * red, k * n, m * n)
    assert ctx.status_poll() == 0
    want = torch.full((groups, n, m), 0.5 * k * red, device="cuda")
    want[1, :, 0] = float("inf")
    assert torch.equal(c.view_as(want), want)


# a sum of a million halves by steps, in one slice and in many; every form that the CUDA cores had
@pytest.mark.parametrize("path", [0, 2, 4])
@pytest.mark.parametrize("m,n,k,red", [(40, 24, 61, 16384), (40, 24, 1000003, 1), (200, 8, 500000, 1), (130, 200, 61, 8192), (136, 264, 999, 1024)])
def test_long_half_sums_have_no_bias(ctx, path, m, n, k, red):
    """Sums of positive halves that TMA cannot address, or of thin products, are as good as fp32 sums rounded to half
    once.  Each result is then off by at most 2^-11 of itself; the mean of these errors, one per output, is zero
    but for 2^-11 / sqrt(3 outputs), and fp32 sums add some 1e-5: their own truncation and promotion."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(9)
    a, b = (torch.rand(red * s, device="cuda", generator=gen).mul_(2.0 ** -7).half() for s in (m * k, k * n))
    c = torch.empty(m * n, device="cuda", dtype=torch.half)
    ctx.gemm(MODES["fp16"], 0, 0, a.data_ptr(), b.data_ptr(), c.data_ptr(), m, n, k, 1, red, 0, m * k, 0, k * n, 0, False, path)
    assert ctx.status_poll() == 0
    a, b = a.view(red, k, m), b.view(red, n, k)
    want = sum(torch.einsum("rkm,rnk->nm", a[i:i + 64].double(), b[i:i + 64].double()) for i in range(0, red, 64))
    off = (c.view(n, m).double() / want - 1).flatten()
    assert off.mean().abs() <= 4 * 2.0 ** -11 / (3 * m * n) ** 0.5 + 1e-5
    assert off.abs().max() <= 2.0 ** -11 + 3e-5


@pytest.mark.parametrize("mode", ["3xtf32", "tf32", "fp16"])
def test_bits_do_not_depend_on_the_plane_cache(ctx, mode):
    """Forward and backward with no planes held, with all that the plane kernels would keep, and with the cache off:
    the same bits.  Sums of more than 1024 terms below 2^32 multiply-adds, whose order the kernels choose themselves."""
    kind = torch.float16 if mode == "fp16" else torch.float32
    gen = torch.Generator(device="cuda")
    gen.manual_seed(2)
    try:
        for di, dj, dk, n in ((1024, 1536, 512, 1), (256, 2048, 256, 1), (515, 1100, 387, 2), (256, 1300, 1024, 3), (2048, 1111, 333, 1), (700, 1600, 900, 1)):
            a, b, gy = (torch.randn(n * s, device="cuda", generator=gen).to(kind) for s in (di * dj, dj * dk, di * dk))
            y, ga, gb = torch.empty_like(gy), torch.empty_like(a), torch.empty_like(b)

            def step():
                ctx.matmul_fw(MODES[mode], a.data_ptr(), b.data_ptr(), y.data_ptr(), di, dj, dk, n, n)
                ctx.matmul_bw_ex(MODES[mode], a.data_ptr(), b.data_ptr(), gy.data_ptr(), ga.data_ptr(), gb.data_ptr(), di, dj, dk, n, n, False, False)
                return [x.clone() for x in (y, ga, gb)]

            ctx.operand_cache_enable(0)
            off = step()
            ctx.operand_cache_enable(1 << 30)
            cold = step()
            ctx.set_path_policy(2)      # every product by planes: they are all held afterwards
            step()
            ctx.set_path_policy(0)
            held = step()
            for x, others in zip(off, zip(cold, held)):
                assert all(torch.equal(x, o) for o in others), (di, dj, dk, n)
    finally:
        ctx.set_path_policy(0)
        ctx.operand_cache_enable(0)


@pytest.mark.parametrize("layout", ["nn", "tn"])
def test_non_finite_sums_are_mended_everywhere(ctx, layout):
    """Every output infinite, at ragged ends of the tiles, with slices, and with operands exchanged; and in the time that
    the CUDA cores take, measured 1.2 and 0.7 of it (a chain of single elements per thread: 8.5 and 2.7)."""
    ta, tb = (int(c == "t") for c in layout)
    for m, n, k in ((131, 9, 1100), (9, 131, 1100), (70, 15, 40), (1030, 8, 4099)):
        a, b = torch.full((m * k,), float("inf"), device="cuda"), torch.full((k * n,), 0.5, device="cuda")
        for mode in ("3xtf32", "tf32", "3xfp16"):
            c = torch.full((m * n + 4,), 7.0, device="cuda")
            ctx.gemm(MODES[mode], ta, tb, a.data_ptr(), b.data_ptr(), c.data_ptr(), m, n, k, force_path=4)
            assert ctx.status_poll() == 0
            assert torch.isposinf(c[:m * n]).all() and (c[m * n:] == 7.0).all(), (m, n, k, mode)
    m, n, k = 64, 8, 65536
    a, b, c = torch.full((m * k,), float("nan"), device="cuda"), torch.ones(k * n, device="cuda"), torch.empty(m * n, device="cuda")

    def us(path):
        best = []
        for _ in range(5):
            start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            start.record()
            ctx.gemm(MODES["3xtf32"], ta, tb, a.data_ptr(), b.data_ptr(), c.data_ptr(), m, n, k, force_path=path)
            end.record()
            end.synchronize()
            best.append(start.elapsed_time(end) * 1e3)
        return min(best)

    assert us(4) <= 2 * us(1)
