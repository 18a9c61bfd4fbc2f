"""The order by length of causal items (attn_sched.cuh: fa_length_rank; the kByLen kernels of
fa_fwd_sm100.cu): the header's own function compiled on the host, the choice between this
order and pairs or a cut through ptxb200_fa_plan_ex, and on the GPU the same bits as with
single blocks dealt round robin."""
import ctypes
import os
import subprocess

import pytest
import torch

from test_attention_tail_split import item_steps, plan as round_robin_plan, unit_items

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MIB = 1 << 20


@pytest.fixture(scope="module")
def ranks(tmp_path_factory):
    """(grid, items) -> each CTA's places in the order by length."""
    exe = str(tmp_path_factory.mktemp("sched") / "attn_sched_dump")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "ptx.jl_b200", "csrc"),
                    os.path.join(ROOT, "tests", "host", "attn_sched_dump.cpp"), "-o", exe], check=True)

    def run(grid, items):
        out = subprocess.run([exe, str(grid), str(items)], check=True, stdout=subprocess.PIPE, text=True).stdout
        return [[int(r) for r in line.split()] for line in out.splitlines()]

    return run


def plan(pkg, B, H, H_kv, S, D, causal=True, flags=0, sm=148):
    cap = 16 + sm * 49
    buf = (ctypes.c_int * cap)()
    n = pkg.native.lib().ptxb200_fa_plan_ex(B, H, H_kv, S, D, int(causal), flags, sm, buf, cap)
    assert n >= 11, n
    keys = ["nmb", "bh", "nt_all", "causal", "pair", "grid", "full", "tail_units", "tail_steps", "tail_ctas", "by_length"]
    return dict(zip(keys, buf[:11])), n


@pytest.mark.parametrize("bh,nmb", [(1, 149), (32, 12), (32, 8), (64, 4), (36, 6), (149, 1), (7, 64), (512, 2)])
def test_every_item_once_and_evenly(ranks, bh, nmb):
    grid, nt_all = 148, 2 * nmb
    steps = lambda mb: min(2 * mb + 2, nt_all)
    seen, loads = [], []
    for mine in ranks(grid, bh * nmb):
        mine = [(nmb - 1 - r // bh, r % bh) for r in mine]
        assert [m for m, _ in mine] == sorted((m for m, _ in mine), reverse=True)   # longest first
        seen += mine
        loads.append(sum(steps(m) for m, _ in mine))
    assert len(loads) == grid
    assert sorted(seen) == sorted((m, h) for m in range(nmb) for h in range(bh))
    # lengths fall by at most one block's two steps from rank to rank within a level change, so
    # going to and fro leaves no CTA more than the longest item above the mean
    assert max(loads) <= sum(loads) / grid + steps(nmb - 1)


def test_choice_of_the_order_by_length(pkg):
    n = pkg.native
    p, ints = plan(pkg, 1, 32, 8, 3001, 128)
    assert p["by_length"] == 1 and p["pair"] == 0 and p["tail_units"] == 0 and ints == 11
    assert p["grid"] == 148 and p["full"] == 32 * 12
    # flags that ask for another distribution, and launches without masks
    assert plan(pkg, 1, 32, 8, 3001, 128, flags=n.FA_SINGLE_BLOCKS)[0]["by_length"] == 0
    assert plan(pkg, 1, 32, 8, 3001, 128, flags=n.FA_ALWAYS_TAIL_SPLIT)[0]["by_length"] == 0
    assert plan(pkg, 1, 32, 8, 3001, 128, causal=False)[0]["by_length"] == 0
    # no more items than SMs: nothing to deal
    assert plan(pkg, 1, 148, 4, 256, 128)[0]["by_length"] == 0
    # K and V of all heads up to 160 MiB: 5 x 32 heads of 2048 keys are exactly that at head dim 128
    assert 4 * 5 * 32 * 2048 * 128 == 160 * MIB
    assert plan(pkg, 5, 32, 32, 2048, 128)[0]["by_length"] == 1
    assert plan(pkg, 5, 32, 32, 2049, 128)[0]["by_length"] == 0
    assert plan(pkg, 5, 32, 32, 2049, 64)[0]["by_length"] == 1
    assert plan(pkg, 5, 32, 8, 2049, 128)[0]["by_length"] == 1


def test_choice_beats_round_robin_by_three_percent(pkg, ranks):
    """Taken when the busiest CTA's steps, one more for each item boundary, are at least 3 % below
    those of the pairs or single blocks dealt round robin that ptxb200_fa_plan shows."""
    choices = set()
    for bh, nmb in [(32, 12), (32, 8), (64, 4), (36, 6), (48, 5), (16, 20), (150, 1), (148, 2), (74, 4), (37, 8), (296, 3),
                    (592, 2), (444, 5), (148, 9)]:
        nt_all = 2 * nmb
        busiest = max(sum(min(2 * (nmb - 1 - r // bh) + 2, nt_all) + 1 for r in mine) for mine in ranks(148, bh * nmb))
        sc, _ = round_robin_plan(pkg, bh, 256 * nmb, True, pkg.native.FA_NO_TAIL_SPLIT)
        loads = [0] * 148
        for q in range(sc["full"]):
            loads[q % 148] += sum(item_steps(mb, nt_all, True) for mb, _ in unit_items(sc, q))
        boundaries = 2 * -(-sc["full"] // 148) if sc["pair"] else -(-bh * nmb // 148)
        want = busiest * 100 <= (max(loads) + boundaries) * 97
        assert plan(pkg, 1, bh, 1, 256 * nmb, 64, flags=pkg.native.FA_NO_TAIL_SPLIT)[0]["by_length"] == want, (bh, nmb)
        choices.add(want)
    assert choices == {False, True}


def test_plan_ex_arguments(pkg):
    n, f = pkg.native, pkg.native.lib().ptxb200_fa_plan_ex
    buf = (ctypes.c_int * 16)()
    assert f(1, 32, 8, 3001, 128, 1, 0, 148, buf, 10) == n.E_CAPACITY
    assert f(1, 32, 0, 3001, 128, 1, 0, 148, buf, 16) == n.E_INVALID
    assert f(1, 32, 5, 3001, 128, 1, 0, 148, buf, 16) == n.E_SHAPE
    assert f(1, 32, 8, 3001, 96, 1, 0, 148, buf, 16) == n.E_SHAPE
    assert f(1, 32, 8, 3001, 128, 2, 0, 148, buf, 16) == n.E_INVALID


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
    sm = torch.cuda.get_device_properties(gpu).multi_processor_count
    assert plan(pkg, B, H, H_kv, S, D, flags=pkg.native.FA_NO_TAIL_SPLIT, sm=sm)[0]["by_length"] == 1
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
