"""Block order of the attention launches (csrc/attn/work_order.h) on the CPU, and the backward kernels at the edges of
their tiles, item counts and output forms on a GPU."""
import math

import pytest
import torch

from zenyx_b200.ops import _ext
from zenyx_b200.ops.attention import MaskSpec, attn_backward, attn_forward, flash_attention, ring_flash_attention


@pytest.mark.parametrize("n_tiles", [1, 2, 3, 17, 64, 256, 300])
@pytest.mark.parametrize("n_heads", [1, 3, 8, 32])
@pytest.mark.parametrize("uniform,everything", [(False, False), (True, False), (False, True)])
def test_block_order_takes_every_tile_of_every_head_once(n_tiles, n_heads, uniform, everything):
    per, order = _ext.host().attn_work_order(n_tiles, n_heads, n_tiles, uniform, everything)
    assert 1 <= per <= n_heads
    assert sorted(order) == [(t, h) for t in range(n_tiles) for h in range(n_heads)]
    groups = [order[i: i + n_tiles * per] for i in range(0, len(order), n_tiles * per)]
    for g, blocks in enumerate(groups):
        assert [t for t, _ in blocks] == sorted(t for t, _ in blocks)             # longest first inside a group
        assert {h for _, h in blocks} == set(range(g * per, min(n_heads, (g + 1) * per)))


@pytest.mark.gpu
@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("B,Sq,Skv,Hq,Hkv,causal,wb,ge,qpos,kpos", [
    (1, 128, 128, 1, 1, True, 0, 0, [0], [0]),                  # one item, one block
    (2, 128, 256, 2, 1, False, 0, 0, [0], [0]),                 # two items per block: every stage used once
    (1, 640, 640, 3, 3, True, 0, 0, [0], [0]),                  # 1 to 5 items: all stage counts wrap
    (1, 512, 768, 4, 2, True, 0, 0, [0, 1024], [256, 896, 512]),   # unsorted chunks; tiles that see and are seen by nothing
    (1, 1024, 1024, 2, 1, True, 2, 3, [0], [0]),                # window and global tiles
])
def test_attention_backward_writes_every_tile(B, Sq, Skv, Hq, Hkv, causal, wb, ge, qpos, kpos, bf16):
    """The written (not accumulated) gradients, fp32 and bf16, against the fp32 host path. The buffers start as NaN: a
    tile without work has to be written too. Bound: P and dS are rounded to bf16 (2^-9 each) before products whose
    terms partly cancel; the accumulating form of the same kernels is held to 2e-2 in test_gpu_kernels.py."""
    torch.manual_seed(Sq + Skv)
    mask, scale = MaskSpec(causal, wb, ge), 1.0 / math.sqrt(128)
    q, do = (torch.randn(B, Sq, Hq, 128).bfloat16() for _ in range(2))
    k, v = (torch.randn(B, Skv, Hkv, 128).bfloat16() for _ in range(2))
    results = []
    for dev in ("cpu", "cuda"):
        a = [t.to(dev) for t in (q, k, v, do)]
        o, lse = torch.empty_like(a[0]), torch.empty(B, Hq, Sq, device=dev)
        attn_forward(a[0], a[1], a[2], o, lse, scale, mask, qpos, kpos)
        grads = [torch.full(t.shape, math.nan, device=dev, dtype=torch.bfloat16 if bf16 and dev == "cuda" else torch.float32)
                 for t in (q, k, v)]
        attn_backward(*a[:3], o, a[3], lse, torch.empty_like(lse), *grads, scale, mask, qpos, kpos, kv_overwrite=True)
        results.append([g.float().cpu() for g in grads])
    _ext.check_status()
    for ref, got in zip(*results):
        assert torch.isfinite(got).all()
        assert (got - ref).norm() <= 2e-2 * ref.norm()
        # Zero rows: nothing seen, or (window case, row 0) one key, where dP - delta is the difference of two 32-bit sums
        # of 128 products of unit normals, each off by at most 128 * 2^-24 * sum|terms| ~ 1e-3 * 2^-7 ~ 1e-5.
        assert got[ref.abs().amax(-1) == 0].abs().amax().item() <= 1e-5 if (ref.abs().amax(-1) == 0).any() else True


@pytest.mark.gpu
@pytest.mark.parametrize("gain", [1.0, 12.0])
@pytest.mark.parametrize("B,Sq,Skv,Hq,Hkv,causal,wb,ge,qpos,kpos", [
    (1, 128, 128, 1, 1, True, 0, 0, [0], [0]),              # one Q tile: the second half of the block has nothing to do
    (2, 384, 640, 2, 1, False, 0, 0, [0], [0]),             # odd tile counts
    (1, 768, 1536, 2, 2, True, 0, 0, [0, 1152], [0]),       # a pair of Q tiles across two chunks: 3 and 10 KV tiles
    (1, 768, 768, 2, 1, True, 0, 0, [1152, 0], [768, 0]),   # the other way round, and a tile that sees nothing at first
    (1, 1280, 1280, 1, 1, True, 2, 4, [0], [0]),            # window and global tiles
])
def test_attention_forward_pairs_and_rescaling(B, Sq, Skv, Hq, Hkv, causal, wb, ge, qpos, kpos, gain):
    """One call, and two calls over the halves of the keys merged, against the fp32 host path. `gain` makes the row maxima
    grow from tile to tile by more than the 2^8 that the kernel tolerates, so the output is rescaled in flight. Bound:
    P and V are rounded to bf16 (2^-9), the merged form rounds the output to bf16 twice."""
    torch.manual_seed(Sq + Skv)
    mask, scale = MaskSpec(causal, wb, ge), gain / math.sqrt(128)
    q = torch.randn(B, Sq, Hq, 128).bfloat16()
    k, v = (torch.randn(B, Skv, Hkv, 128).bfloat16() for _ in range(2))
    half = Skv // (2 * len(kpos)) * len(kpos) if Skv % (256 * len(kpos)) == 0 else 0
    results = []
    for dev in ("cpu", "cuda"):
        a = [t.to(dev) for t in (q, k, v)]
        out = []
        for merge in ([False, True] if half and len(kpos) == 1 else [False]):
            o = torch.full(q.shape, math.nan, device=dev, dtype=torch.bfloat16)
            lse = torch.full((B, Hq, Sq), math.nan, device=dev)
            if merge:
                lo, hi = ([t[:, part].clone(memory_format=torch.contiguous_format) for t in a[1:]]
                          for part in (slice(0, half), slice(half, None)))
                attn_forward(a[0], *hi, o, lse, scale, mask, qpos, [half])
                attn_forward(a[0], *lo, o, lse, scale, mask, qpos, [0], True)
            else:
                attn_forward(*a, o, lse, scale, mask, qpos, kpos)
            out += [o.float().cpu(), lse.cpu()]
        results.append(out)
    _ext.check_status()
    for n, (ref, got) in enumerate(zip(*results)):
        if n % 2 == 0:
            assert torch.isfinite(got).all()
            assert (got - ref).norm() <= 2e-2 * ref.norm()
        else:
            seen = torch.isfinite(ref)
            assert torch.equal(seen, torch.isfinite(got))
            # scores are exact products summed in fp32: |s| up to ~60 with the gain, 128 terms, plus the exponentials' 2^-22
            assert (got[seen] - ref[seen]).abs().max().item() <= 2e-3


def _shifted(t, elements):
    """A contiguous copy of t that starts `elements` elements into a 16-byte unit."""
    buf = torch.empty(t.numel() + 8, device=t.device, dtype=t.dtype)
    out = buf[elements: elements + t.numel()].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.gpu
def test_attention_backward_takes_o_at_8_bytes_and_refuses_before_it_launches():
    """o is read by the delta pre-pass alone, 8 bytes of it at the least; d_o by TMA too, which takes 16-byte units."""
    torch.manual_seed(5)
    B, S, Hq, Hkv, scale = 2, 256, 4, 2, 1.0 / math.sqrt(128)
    q, do = (torch.randn(B, S, Hq, 128, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(B, S, Hkv, 128, device="cuda").bfloat16() for _ in range(2))
    o, lse = torch.empty_like(q), torch.empty(B, Hq, S, device="cuda")
    attn_forward(q, k, v, o, lse, scale, MaskSpec(), [0], [0])

    def backward(o, do):
        delta = torch.full_like(lse, 7.0)
        grads = [torch.full(t.shape, 7.0, device="cuda") for t in (q, k, v)]
        try:
            attn_backward(q, k, v, o, do, lse, delta, *grads, scale, MaskSpec(), [0], [0], kv_overwrite=True)
        except RuntimeError as e:
            assert "aligned" in str(e)
            assert all((t == 7.0).all() for t in (delta, *grads))   # nothing ran
            return None
        return (delta, *grads)

    want = backward(o, do)
    got = backward(_shifted(o, 4), do)
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    for elements in (1, 2):
        assert backward(_shifted(o, elements), do) is None
    for elements in (1, 4):
        assert backward(o, _shifted(do, elements)) is None
    _ext.check_status()


def test_gradients_of_mixed_types_are_rounded_to_each_input_s_own():
    """A ring of one rank on the CPU takes q, k and v of different types; fp32 gradients are not rounded to q's type."""
    torch.manual_seed(6)
    q = torch.randn(1, 128, 2, 128).bfloat16().requires_grad_(True)
    k, v = (torch.randn(1, 128, 1, 128).requires_grad_(True) for _ in range(2))
    do = torch.randn(1, 128, 2, 128).bfloat16()
    got = torch.autograd.grad(ring_flash_attention(q, k, v), (q, k, v), do)
    want = torch.autograd.grad(flash_attention(q, k, v), (q, k, v), do)
    assert [g.dtype for g in got] == [torch.bfloat16, torch.float32, torch.float32]
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def _row_sum_noise(heads=8, rows=256, keys=131072):
    """Root mean square error of the log-sum-exp over rows, less each head's mean. One key has score 0 and comes first (no
    rescaling), the others about -6.5: the scores are exact in fp32, the row sum is about 200, the log-sum-exp about 5, so
    that little but the additions of the row sum is left to be wrong."""
    torch.manual_seed(7)
    q, k = torch.zeros(1, rows, heads, 128, device="cuda"), torch.zeros(1, keys, heads, 128, device="cuda")
    q[..., 0] = (64 + torch.arange(rows, device="cuda") % 64)[None, :, None] / 256
    q[..., 1] = 6.9375
    k[..., 0] = torch.rand(1, keys, heads, device="cuda").add_(1).mul_(0.5)
    k[..., 1] = -1
    k[:, 0] = 0
    q, k = q.bfloat16(), k.bfloat16()
    o, lse = torch.empty_like(q), torch.empty(1, heads, rows, device="cuda")
    attn_forward(q, k, k, o, lse, 1.0, MaskSpec(False), [0], [0])
    _ext.check_status()
    err = torch.empty_like(lse, dtype=torch.float64)
    for h in range(heads):
        err[0, h] = lse[0, h].double() - torch.logsumexp(q[0, :, h, :2].double() @ k[0, :, h, :2].double().T, -1)
    return (err - err.mean(-1, keepdim=True)).square().mean().sqrt().item()


@pytest.mark.gpu
def test_row_sums_are_rounded_at_their_own_magnitude_once_per_half_tile():
    """131,072 keys: 2,048 halves of 64 keys, whose sums each thread adds to a running sum of its even and one of its odd
    columns. Rounding to nearest at the running value (standard deviation 0.29 * 2^-23.5 of it, on average over its growth
    0.58 of the final one) 2,048 times in each of the eight running sums of a row: 45 * 2.4e-8 * 0.58 / sqrt(8) = 2.2e-7 of
    the row sum, the logarithm's own rounding about 1e-7. Measured: 3.0e-7, and 5.9e-6 with the terms added to the running sum one
    by one."""
    assert _row_sum_noise() <= 5e-7
