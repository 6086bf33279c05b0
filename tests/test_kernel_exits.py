"""Waits that give up must not strand anybody at a barrier. The kernels' waits are bounded, a warp whose wait runs out leaves its loop; where several warps
meet in that loop, it owes the others the meetings that are left. Checked by counting, with the expressions of the source: a run in which a wait fails
is no test for a shared GPU."""
import re
from pathlib import Path

TEXT = (Path(__file__).resolve().parent.parent / "oxinfer_b200" / "csrc" / "gemv_tc.cu").read_text()
ROLE = TEXT[TEXT.index("if (warp > 1) {"):TEXT.index("} else if (warp == 0) {")]


def the(pattern):
    found = re.findall(pattern, ROLE)
    assert len(found) == 1, (pattern, found)
    return found[0]


def test_a_warp_that_leaves_its_set_meets_it_as_often_as_the_set_does():
    meets, share = the(r"const int meets = MEETS \* (.*);"), the(r"const int share = (.*);")
    assert the(r"for \(int lb = (share; lb < nbq && ok; lb \+= GT_SETS)\)")
    whole_tiles = the(r"if constexpr \(MLX\) met = (\(i .*);")
    for nbq in range(0, 42):
        for tiles in range(0, 9):
            for s in range(4):
                blocks = sum(len(range(eval(share, {"set": s, "i": i, "nbq": nbq}), nbq, 4)) for i in range(tiles))
                assert blocks == eval(meets, {"total": tiles * nbq, "set": s}), (nbq, tiles, s)
                assert tiles == 0 or blocks == eval(whole_tiles, {"i": tiles - 1, "nbq": nbq, "set": s})
    # and the blocks of block n's set (n % 4) ahead of it
    assert the(r"if constexpr \(MLX\) met = (n .*);") == "n >> 2" and "met = (n >> 2) + 1;" in ROLE


def test_every_meeting_is_counted_and_the_rest_is_made_up_for():
    code = re.sub(r"//[^\n]*", "", ROLE)
    # one barrier in the loop, counted, and one that makes up for the meetings that are left, behind it
    barriers = [m.start() for m in re.finditer(r"bar\.sync", code)]
    assert len(barriers) == 2 and code[barriers[0]:].split("\n")[1].strip() == "if constexpr (!MLX) met++;"
    assert re.search(r"if \(!ok\) \{[^{}]*const int meets = [^;]*;\s*for \(; met < meets; met\+\+\) asm", code)
    # MEETS is what a block's path goes through: Q4_K twice, MLX-4 once, Q8_0 eight chunks of 32 values by CHUNKS
    q8, mlx, q4 = (code.index(s) for s in ("if constexpr (Q8) {  ", "} else if constexpr (MLX) {  ", "auto scaled = "))
    assert code[q8:mlx].count("multiply(") == 1 and code[mlx:q4].count("multiply(") == 1 and code[q4:].count("multiply(") == 2
    assert "k0 < 8; k0 += CHUNKS" in code and "CHUNKS = NB == 16 ? 8 : 4" in code
    assert the(r"constexpr int MEETS = (.*);") == "MLX || (Q8 && NB == 16) ? 1 : 2"


def test_what_peers_store_is_acquired_at_cluster_scope_and_given_back_after_every_lane_has_read_it():
    """(Read from the source too: on one machine a missing order shows once in a great while.)"""
    attend = (Path(__file__).resolve().parent.parent / "oxinfer_b200" / "csrc" / "attend.cu").read_text()
    for bar in ("in_full[buf]", "in_free[to][buf]", "ssq_full"):  # (counted by the cluster's other CTAs)
        waits = re.findall(r"gt_wait(<true>)?\(&sh->" + re.escape(bar), TEXT)
        assert waits and all(waits), bar
    assert "bar_wait<true>(all_in" in attend and "bar_wait(all_in" not in attend
    give_back = TEXT[TEXT.index("uint32_t words = __float_as_uint(v[0]);"):TEXT.index("gt_arrive(cluster_addr(&sh->in_free[rank][buf]")]
    assert "for (int t = 1; t < TP; t++) words |=" in give_back and re.search(r"words = __(ballot|reduce_or)_sync\(0xffffffffu, words[^;]*\) & \(uint32_t\)a\.zero;", give_back)
