"""The sizes and rules that gemm_split_sm100.cu runs by, from its own header compiled on the
host: every step of K once, chains of at most eight steps, shared and tensor memory within
what an SM has, a slot of its own for everything one CTA of a cluster hands another."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def dump(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("plan") / "gemm_plan_dump")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "ptx.jl_b200", "csrc"),
                    os.path.join(ROOT, "tests", "host", "gemm_plan_dump.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, stdout=subprocess.PIPE, text=True).stdout
    return [line.split() for line in out.strip().splitlines()]


def layouts(dump):
    names = "bn split kiters f32 longest stages chain fold tmem smem recv per".split()
    for line in dump:
        if line[0] == "layout":
            values = list(map(int, line[1:]))
            l = dict(zip(names, values))
            cuts, cols = values[len(names):][:l["split"] + 1], values[len(names):][l["split"] + 1:]
            yield dict(l, cuts=cuts, cols=cols)


def test_parts_cover_k_once_and_chains_are_short(dump):
    n = 0
    for l in layouts(dump):
        cuts, bn, per = l["cuts"], l["bn"], l["per"]
        assert cuts[0] == 0 and cuts[-1] == l["kiters"] and len(cuts) == l["split"] + 1
        for a, b in zip(cuts, cuts[1:]):
            assert b > a                                        # no part without a step
            ring = -(-(b - a) // per)                           # stages this part fills
            chains = -(-ring // l["chain"])
            if l["longest"] == 0:
                assert chains == 1                              # one accumulation in k order
            else:                                               # never above what the caller allows, or 8
                assert l["chain"] * per <= max(8, l["longest"]) or chains == 1 and b - a <= max(8, l["longest"])
            most = -(-max(y - x for x, y in zip(cuts, cuts[1:])) // 8)     # chains of 8 that the longest part takes
            if l["f32"] and l["longest"] and (l["split"] == 1 or most * bn <= 512):
                assert l["chain"] * per <= 8                    # longer only where accumulators run out
            # accumulators: two in turn, with another for what they add up to where K is split, or all
            blocks = 3 if l["fold"] else min(chains, 2) if l["split"] == 1 else chains
            if bn == 192 and l["fold"]:
                continue                                        # 192 columns have no third block: see the rule's test
            assert bn * blocks <= l["tmem"] <= 512 and l["tmem"] & (l["tmem"] - 1) == 0
        n += 1
    assert n > 1000


def test_memory_fits_and_clusters_do_not_share_an_sm(dump):
    for l in layouts(dump):
        assert 1 <= l["stages"] <= 7
        ring = l["stages"] * l["per"] * (128 + l["bn"]) * 128
        assert ring + 160 + l["recv"] <= l["smem"] <= 232448
        if l["split"] > 1:
            assert 2 * (l["smem"] + 1024) > 233472              # an SM's 228 KiB


@pytest.mark.parametrize("bn,split", [(64, 2), (64, 4), (128, 2), (128, 3), (128, 4), (128, 5), (128, 6), (128, 8), (192, 2)])
def test_each_pair_of_parts_has_a_slot_of_its_own(dump, bn, split):
    """The kernel's indexing: sender p's 16-byte pieces of the columns that q sums up go to slot
    (p < q ? p : p - 1) of q, [columns / 4][128 rows] of them; the shares cover the tile once."""
    l = next(l for l in layouts(dump) if l["bn"] == bn and l["split"] == split)
    cols, slot_bytes = l["cols"], l["recv"] // (split - 1)
    assert cols[0] == 0 and cols[-1] == bn and len(cols) == split + 1
    assert all(b > a and a % 16 == 0 for a, b in zip(cols, cols[1:]))
    for q in range(split):
        seen = set()
        for p in range(split):
            if p == q:
                continue
            slot = p if p < q else p - 1
            for c in range(0, cols[q + 1] - cols[q], 16):
                for j in range(4):
                    for row in range(128):
                        seen.add(slot * slot_bytes + (c // 4 + j) * (128 * 16) + row * 16)
        assert len(seen) == (split - 1) * 128 * (cols[q + 1] - cols[q]) // 4
        assert min(seen) == 0 and max(seen) + 16 <= l["recv"]


def test_rule_runs_every_cluster_at_once(dump):
    rules = [list(map(int, line[1:])) for line in dump if line[0] == "rule"]
    assert len(rules) == 3 * 2 * 300 * 10 * 2
    used = set()
    for set_, rows, n, kiters, may, here, bn, split, clusters, fold, tmem in rules:
        tiles128 = rows * ((n + 1) // 2)
        assert bool(here) == (tiles128 <= 148)
        if not here:
            continue
        tiles = rows * -(-n // (bn // 64))
        assert tiles * split <= 148 and split <= kiters
        assert split == 1 or may and kiters >= 16
        assert split <= 2 or tiles <= clusters      # clusters do not fill all SMs: 33 of 37 of four fit
        assert bn < 192 or split == 2 and not fold and tmem <= 512
        used.add((bn, split))
    assert used == {(64, 1), (64, 2), (64, 4), (128, 1), (128, 2), (128, 3), (128, 4), (128, 5), (128, 6), (128, 8), (192, 2)}
    split = lambda n, k, c: next(r[6:8] for r in rules if r[:5] == [c, 1, n, k, 1])
    assert [split(n, 64, 1)[1] for n in (32, 33, 34, 37, 74)] == [4, 4, 2, 2, 2]
    assert split(75, 16, 1) == [64, 1] and split(75, 64, 1) == [128, 2]
    assert split(30, 192, 1) == [128, 8] and split(31, 192, 1) == split(33, 192, 1) == [64, 4]
    assert split(34, 192, 1) == [128, 6] and split(90, 192, 1) == [128, 3]
    assert split(91, 192, 1) == [128, 2] and split(149, 192, 1) == [192, 2] and split(149, 191, 1) == [128, 1]
    assert split(223, 192, 1) == [128, 1]


def test_shares_of_one_line_of_steps(dump):
    """What bounds the chains of sums: at most half as many 128x256 tiles as SMs, shares of at
    least eight steps, two shares or more per tile; otherwise all of K."""
    n = 0
    for tiles, kiters, ctas, share in (map(int, line[1:]) for line in dump if line[0] == "line"):
        want = min(tiles * kiters // 8, 148)
        if tiles > 74 or want < 2 * tiles:
            assert (ctas, share) == (0, kiters)
        else:
            assert ctas == want and 8 <= share == -(-tiles * kiters // ctas) < kiters
            n += 1
    assert n > 20
    line = {(int(l[1]), int(l[2])): (int(l[3]), int(l[4])) for l in dump if l[0] == "line"}
    assert line[(1, 128)] == (16, 8) and line[(32, 128)] == (148, 28) and line[(75, 128)] == (0, 128)
