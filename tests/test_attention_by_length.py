"""The order by length of causal items (attn_sched.cuh: fa_length_rank; the kByLen kernels of
fa_fwd_sm100.cu): a CPU model of who runs what, and on the GPU the same bits as with single
blocks dealt round robin."""
import itertools

import pytest
import torch


def rank(cta, v, grid):
    return v * grid + (grid - 1 - cta if v & 1 else cta)


def items_of(cta, grid, bh, nmb):
    out = []
    for v in itertools.count():
        r = rank(cta, v, grid)
        if r >= bh * nmb:
            return out
        out.append((nmb - 1 - r // bh, r % bh))


@pytest.mark.parametrize("bh,nmb", [(1, 149), (32, 12), (32, 8), (64, 4), (36, 6), (149, 1), (7, 64), (512, 2)])
def test_every_item_once_and_evenly(bh, nmb):
    grid, nt_all = 148, 2 * nmb
    steps = lambda mb: min(2 * mb + 2, nt_all)
    seen, loads = [], []
    for cta in range(grid):
        mine = items_of(cta, grid, bh, nmb)
        assert [m for m, _ in mine] == sorted((m for m, _ in mine), reverse=True)   # longest first
        seen += mine
        loads.append(sum(steps(m) for m, _ in mine))
    assert sorted(seen) == sorted((m, h) for m in range(nmb) for h in range(bh))
    # lengths fall by at most one block's two steps from rank to rank within a level change, so
    # going to and fro leaves no CTA more than the longest item above the mean
    assert max(loads) <= sum(loads) / grid + steps(nmb - 1)


@pytest.mark.gpu
@pytest.mark.parametrize("B,H,H_kv,S,D,lse", [
    (1, 32, 8, 2048, 128, False),   # two rounds
    (1, 32, 8, 1501, 128, True),    # a last block that is only partly there, odd tile count
    (6, 8, 8, 900, 128, True),
    (20, 16, 16, 300, 128, False),  # two blocks a head
    (1, 150, 50, 129, 64, True),    # one block a head, two more items than CTAs
    (2, 24, 8, 1700, 64, False),
])
def test_same_bits_as_round_robin(pkg, gpu, B, H, H_kv, S, D, lse):
    g = torch.Generator(device=gpu).manual_seed(S + D)
    q = torch.randn(B, H, S, D, generator=g, device=gpu).to(torch.bfloat16)
    k, v = (torch.randn(B, H_kv, S, D, generator=g, device=gpu).to(torch.bfloat16) for _ in range(2))
    got, want = torch.full_like(q, float("nan")), torch.full_like(q, float("nan"))
    stats = [torch.empty(B * H * S, device=gpu) if lse else None for _ in range(2)]
    pkg.ops.fa_fwd(q, k, v, causal=True, out=got, lse=stats[0], flags=pkg.native.FA_NO_TAIL_SPLIT)
    pkg.ops.fa_fwd(q, k, v, causal=True, out=want, lse=stats[1],
                   flags=pkg.native.FA_SINGLE_BLOCKS | pkg.native.FA_NO_TAIL_SPLIT)
    status = pkg.ops.sync_status()
    assert status == 0, pkg.native.strerror(status)
    assert torch.equal(got, want)
    assert not lse or torch.equal(*stats)
