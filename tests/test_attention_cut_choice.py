"""When the last round of attention items is cut along the key axis by default (plan_schedule,
fa_fwd_sm100.cu): where the busiest CTA's steps with all that a cut costs -- a base by head dim and a
step per further piece of an item -- stay 3 % below those of whole items."""
import pytest

from test_attention_by_length import plan, ranks  # noqa: F401 (a fixture)
from test_attention_tail_split import FA_ALWAYS, check_plan, item_steps, plan as plan_128, unit_items

FA_NO_TAIL_SPLIT = 0x4


def busiest_whole(pkg, bh, S, causal):
    sc, _ = plan_128(pkg, bh, S, causal, FA_NO_TAIL_SPLIT)
    load = [0] * sc["grid"]
    for q in range(sc["full"]):
        load[q % sc["grid"]] += sum(item_steps(mb, sc["nt_all"], causal) for mb, _ in unit_items(sc, q))
    return max(load)


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D,base", [(128, 8), (64, 6)])
def test_cut_only_where_it_pays(pkg, causal, D, base):
    taken = set()
    for bh in (1, 3, 8, 16, 20, 40):
        for S in (512, 1024, 1500, 2048, 4096, 8192):
            if plan(pkg, 1, bh, bh, S, D, causal, FA_NO_TAIL_SPLIT)[0]["by_length"]:
                continue                    # (another whole distribution to compare with)
            got = plan(pkg, 1, bh, bh, S, D, causal)[0]["tail_units"] > 0
            sc, ctas = plan_128(pkg, bh, S, causal, FA_ALWAYS)
            want = False
            if sc["tail_units"]:
                full = [0] * sc["grid"]
                for q in range(sc["full"]):
                    full[q % sc["grid"]] += sum(item_steps(mb, sc["nt_all"], causal) for mb, _ in unit_items(sc, q))
                tail = max(sum(j1 - j0 for _, _, j0, j1, _, _ in segs) for segs in ctas)
                pieces = max(no for segs in ctas for *_, no in segs)
                whole, cut = busiest_whole(pkg, bh, S, causal), max(full) + tail
                want = (cut + base + pieces) * 100 <= whole * 97 and (cut + 3) * 100 <= whole * 92
                check_plan(sc, ctas)
            assert got == want, (bh, S)
            taken.add(got)
    assert taken == {False, True}


@pytest.mark.parametrize("bh,S,D,causal,cut", [
    (16, 1024, 128, False, False), (12, 1920, 128, False, False), (40, 1024, 128, False, False),   # measured: whole is faster
    (16, 1024, 128, True, False), (4, 2048, 128, False, False),
    (4, 2048, 64, False, True), (2, 8192, 128, False, True), (6, 8192, 64, False, True), (1, 8192, 128, True, True),
])
def test_measured_shapes(pkg, bh, S, D, causal, cut):
    assert (plan(pkg, 1, bh, bh, S, D, causal)[0]["tail_units"] > 0) == cut


@pytest.mark.parametrize("D,base", [(128, 8), (64, 6)])
def test_cut_only_where_it_beats_whole_items_by_length(pkg, ranks, D, base):  # noqa: F811
    """Where whole causal items would be dealt by length, both sides count a step more for every boundary
    between items: the busiest CTA has one per item by length, and two per full round of pairs and
    one ahead of its cut pieces."""
    taken, by_all_costs = set(), 0
    for bh in (5, 6, 10, 12, 16, 20, 40):
        for S in (1700, 2048, 2560, 3001, 3328, 6200, 7566, 8192):
            if not plan(pkg, 1, bh, 1, S, D, True, FA_NO_TAIL_SPLIT)[0]["by_length"]:
                continue
            got = plan(pkg, 1, bh, 1, S, D, True)[0]
            sc, ctas = plan_128(pkg, bh, S, True, FA_ALWAYS)
            n, nt = sc["nmb"], sc["nt_all"]
            whole = max(sum(item_steps(n - 1 - r // bh, nt, True) + 1 for r in mine) for mine in ranks(148, bh * n))
            want = False
            if sc["tail_units"]:
                full = [0] * sc["grid"]
                for q in range(sc["full"]):
                    full[q % sc["grid"]] += sum(item_steps(mb, nt, True) for mb, _ in unit_items(sc, q))
                cut = max(full) + max(sum(j1 - j0 for _, _, j0, j1, _, _ in segs) for segs in ctas)
                cut += (2 if sc["pair"] else 1) * (sc["full"] // 148) + 1
                pieces = max(no for segs in ctas for *_, no in segs)
                least = (cut + 3) * 100 <= whole * 92
                want = (cut + base + pieces) * 100 <= whole * 97 and least
                by_all_costs += least and not want
            assert (got["tail_units"] > 0) == want and got["by_length"] == (not want), (bh, S)
            taken.add(want)
    assert taken == {False, True} and by_all_costs > 2     # all that a cut costs decides where the least of it would not
