"""The GEMM kernels at the edges of their tiles, in every operand layout and output form."""
import pytest
import torch

from zenyx_b200.ops import _ext


@pytest.mark.gpu
@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("M,N,K", [
    (136, 8, 8),        # second half of the tile has 8 rows, one 8-wide column group, one short k-block
    (264, 264, 72),     # one row group and one column group past a tile
    (512, 136, 448),    # exact rows; a remainder of columns; 7 k-blocks
    (2568, 3080, 648),  # several tiles per pair: both accumulators and every stage count wrap
    (4992, 3968, 192),  # 256-wide tiles leave the last wave emptier than 128-wide ones
])
def test_pair_gemm_matches_fp64_in_every_form(M, N, K, a_t, b_t):
    """bf16, bf16 + addend, fp32 and fp32 accumulated in place against an fp64 product of the same operands. The sums are
    fp32 in another order: K terms of |x w| ~ K^-0.5 each, so 1e-5 of the norm; bf16 results add their rounding, 2^-9."""
    torch.manual_seed(M + N + K)
    a = torch.randn((K, M) if a_t else (M, K), device="cuda").bfloat16()
    b = (torch.randn((K, N) if b_t else (N, K), device="cuda") * K ** -0.5).bfloat16()
    ref = (a.t() if a_t else a).double() @ (b if b_t else b.t()).double()
    base = torch.randn(M, N, device="cuda")
    C = _ext.C()

    def run(out, addend=None):
        C.gemm(a, b, out, a_t, b_t, addend)
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
        _ext.C().gemm(a, b, out, False, False, d)
        runs.append(out)
    _ext.check_status()
    assert all(torch.equal(runs[0], r) for r in runs[1:])
    # every element: half a unit in the last place of bf16, and the fp32 sum of K + 1 terms of magnitude up to ~30
    assert ((runs[0].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all()
