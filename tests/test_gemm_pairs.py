"""The GEMM kernels at the edges of their tiles, in every operand layout and output form."""
import pytest
import torch

from zenyx_b200.ops import _ext


@pytest.mark.parametrize("M,N,K,tile", [
    (64, 1024, 1024, 0),        # one row block: half of a pair would be idle
    (8192, 2048, 512, 0),       # short inner dimension
    (8192, 2080, 64, 0),        # (the shapes of the staging slab test below)
    (8192, 2208, 8, 0),
    (256, 2048, 4096, 128),     # too few tiles of 256 columns
    (3000, 2056, 5640, 128),    # a last wave that 256-wide tiles leave emptier
    (4096, 11264, 4096, 256),
    (32768, 28672, 4096, 256),
])
def test_choice_of_the_kernel(M, N, K, tile):
    """The rule on 148 SMs, so that a change of its constants shows which of the tests below lose their kernel."""
    assert _ext.host().gemm_choose_tile(M, N, K, 148) == tile


@pytest.mark.gpu
@pytest.mark.parametrize("tile", [0, 128, 256])   # single CTAs, CTA pairs with tiles of 128 and of 256 columns
@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [
    (136, 8, 8),        # the second CTA of a pair has 8 rows, the pair one 8-wide column group, one short k-block
    (264, 264, 72),     # one row group past a pair's tile, one column group past either width
    (512, 136, 448),    # exact rows; a remainder of columns; 7 k-blocks
    (2568, 3080, 648),  # two to four tiles per pair: both accumulators and every stage count wrap
    (4992, 3968, 192),  # up to nine tiles per pair, three k-blocks each: the epilogue is the longer half
])
def test_gemm_matches_fp64_in_every_form(M, N, K, a_t, b_t, tile):
    """bf16, bf16 + addend, fp32 and fp32 accumulated in place against an fp64 product of the same operands. The sums are
    fp32 in another order: K terms of |x w| ~ K^-0.5 each, so 1e-5 of the norm; bf16 results add their rounding, 2^-9."""
    torch.manual_seed(M + N + K)
    a = torch.randn((K, M) if a_t else (M, K), device="cuda").bfloat16()
    b = (torch.randn((K, N) if b_t else (N, K), device="cuda") * K ** -0.5).bfloat16()
    ref = (a.t() if a_t else a).double() @ (b if b_t else b.t()).double()
    base = torch.randn(M, N, device="cuda")
    C = _ext.C()

    def run(out, addend=None):
        C.gemm(a, b, out, a_t, b_t, addend, tile=tile)
        return out.double()

    def close(got, want, bound):
        assert (got - want).norm() <= bound * want.norm()

    close(run(torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)), ref, 4e-3)
    close(run(torch.empty(M, N, device="cuda", dtype=torch.bfloat16), base.bfloat16()), ref + base.bfloat16().double(), 4e-3)
    close(run(torch.full((M, N), float("nan"), device="cuda")), ref, 1e-5)
    acc = base.clone()
    close(run(acc, acc), ref + base.double(), 1e-5)
    # a window of a larger matrix: nothing outside it changes, whatever the tile hangs over
    big = torch.full((M + 16, N + 64), 7.0, device="cuda")
    view = big[8: M + 8, 32: N + 32]
    close(run(view), ref, 1e-5)
    assert (big[:8] == 7).all() and (big[M + 8:] == 7).all() and (big[:, :32] == 7).all() and (big[:, N + 32:] == 7).all()
    _ext.check_status()


@pytest.mark.gpu
@pytest.mark.parametrize("addend", [False, True])
@pytest.mark.parametrize("N", [2080, 2208])   # the last tile of a row ends after one, after three of four 64-column chunks
@pytest.mark.parametrize("K", [8, 64])        # short: the next tile's accumulator is ready at once
def test_single_cta_epilogue_keeps_its_staging_slabs_apart(N, K, addend):
    """576 single-CTA tiles, so blocks go from a ragged tile to the next one: a slab may only be written again when the
    store that reads it is done. Bits must repeat, and match fp64 within the rounding to bf16 (2^-9 of the norm at most)."""
    torch.manual_seed(N + K)
    M = 8192
    a = torch.randn(M, K, device="cuda").bfloat16()
    b = (torch.randn(N, K, device="cuda") * K ** -0.5).bfloat16()
    d = torch.randn(M, N, device="cuda").bfloat16() if addend else None
    ref = a.double() @ b.double().t() + (d.double() if addend else 0)
    runs = []
    for _ in range(8):
        out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.bfloat16)
        _ext.C().gemm(a, b, out, False, False, d, tile=0)
        runs.append(out)
    _ext.check_status()
    assert all(torch.equal(runs[0], r) for r in runs[1:])
    # every element: half a unit in the last place of bf16, and the fp32 sum of K + 1 terms of magnitude up to ~30
    assert ((runs[0].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all()


@pytest.mark.gpu
def test_accumulation_of_subnormals():
    """The single-CTA kernel adds in registers and takes subnormal operands and results for zero (-ftz); the pair kernel adds
    in L2, where nothing more than that may be lost."""
    M, N, K = 512, 512, 8
    tiny = torch.finfo(torch.float32).tiny   # 2^-126
    a, b = torch.zeros(M, K, device="cuda"), torch.zeros(N, K, device="cuda")
    a[::2, 0] = 2.0 ** -60                   # one product per element: -2^-125, or zero
    b[:, 0] = -(2.0 ** -65)
    a, b = a.bfloat16(), b.bfloat16()
    base = torch.linspace(-4, 4, M * N, device="cuda").view(M, N) * tiny
    want = base.double() + a.double() @ b.double().t()
    results = []
    for tile in (0, 128, 256):
        acc = base.clone()
        _ext.C().gemm(a, b, acc, False, False, acc, tile=tile)
        results.append(acc)
    _ext.check_status()
    assert torch.equal(results[1], results[2])
    assert all((r.double() - want).abs().max().item() <= 2 * tiny for r in results)   # two values below `tiny` taken for zero
