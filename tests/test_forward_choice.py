"""Which kernel a tabular forward takes, against the times of all three (profiles/forward_kernel_choice.csv).  No GPU needed."""
import csv
import ctypes
import os

import pytest

from conftest import ROOT
from hingetreefortorch_b200 import _cabi

KERNELS = ["thread", "tile", "rows"]  # HT_FORWARD_THREADS, _TILES, _ROWS


def forwards():
    with open(os.path.join(ROOT, "profiles", "forward_kernel_choice.csv")) as table:
        for row in csv.DictReader(table):
            sizes = {k: int(row[k]) for k in ("B", "C", "T", "depth", "M", "save")}
            p = _cabi.ForestProblem(_cabi.HT_KIND[row["kind"]], sizes["depth"], sizes["B"], sizes["C"], 1, sizes["T"], sizes["M"],
                                    _cabi.HT_SAVE_FOR_BACKWARD if sizes["save"] else 0, 0)
            row["takes"] = KERNELS[_cabi.library().ht_forest_forward_kernel(ctypes.byref(p))]
            yield row


def test_the_table_says_what_the_library_chooses():
    for row in forwards():
        assert row["takes"] == row["chosen"], row


@pytest.mark.parametrize("column", ["", "_loop"], ids=["cold caches", "in a loop"])
def test_long_and_short_forwards_take_the_kernel_that_costs_less(column):
    """By the time that calls cost, not by their number: together within 1 % of the better kernel, those above 100 us as well, and
    no kind beyond 2.5 % of the better of its two kernels."""
    total = {}
    for row in forwards():
        other = "tile" if row["tile"] else "thread"
        if not row["rows" + column] or not row[other + column]:
            continue
        times = {k: float(row[k + column]) for k in ("rows", other)}
        best = min(times.values())
        for group in (("all",), (other, row["kind"])) + ((("long",),) if best > 100 else ()):
            chosen, least = total.get(group, (0.0, 0.0))
            total[group] = (chosen + times[row["takes"]], least + best)
    ratios = {group: chosen / least for group, (chosen, least) in total.items()}
    assert ratios["all",] < 1.01 and ratios["long",] < 1.01, ratios
    assert max(ratios.values()) < 1.025, ratios


@pytest.mark.parametrize("B,C,T,depth,M", [(3146, 1194, 616, 8, 8), (3334, 1212, 718, 7, 16), (1716, 1173, 791, 7, 16),
                                           (51359, 1541, 701, 7, 1), (44800, 879, 352, 10, 1), (18319, 1879, 305, 8, 1)])
def test_wide_rows_under_many_trees(B, C, T, depth, M):
    """These run 1.3 to 2.0 times as long with a thread per evaluation, their parameters being too many for L1."""
    p = _cabi.ForestProblem(0, depth, B, C, 1, T, M, 0, 0)
    assert KERNELS[_cabi.library().ht_forest_forward_kernel(ctypes.byref(p))] == "rows"
