"""Orders of waits and announcements in the kernels, on a model of the barriers: every interleaving ends, and every wait that
passes means what it is taken for."""
from functools import lru_cache

import pytest


def passes(completed: int, parity: int) -> bool:
    """mbarrier.try_wait.parity: has the phase of that parity completed?  The barrier knows the current phase's parity only."""
    return completed & 1 != parity


@pytest.mark.parametrize("blocks", [(1,), (3,), (1, 1), (2, 1), (1, 2), (3, 2), (1, 1, 1), (2, 1, 1), (1, 1, 1, 1), (2, 3, 1)])
@pytest.mark.parametrize("wait", ["o_full twice", "v_empty"])
def test_last_unit_of_the_gated_cta_pairs(blocks, wait):
    """sdpa_prefill_wide_kernel, GATE: a softmax warp goes on to write columns of its pair's last unit once that unit's last
    P V has landed.  Units of `blocks` key blocks; the issuer computes a block's scores before the P V of the block before,
    which needs the warp's probabilities.  The warp may be late at any point.  (Waiting for o_full of the unit before and then of
    the last one does not end where the last one is complete as well when the first wait is looked at.)"""
    total = sum(blocks)
    last = [sum(blocks[:u + 1]) - 1 for u in range(len(blocks))]  # last block of each unit
    n = len(blocks)

    def o_full(pv):
        return sum(b < pv for b in last)

    def v_empty(pv, stage):
        return (pv + 1 - stage) // 2

    @lru_cache(None)
    def stuck(scores, pv, said, step):
        """Scores and P V completed, blocks announced; step: waits passed behind the last announcement.  Does some order not end?"""
        moves = []
        if scores < total and pv >= scores - 1:  # S(b) behind P V (b - 2) in the tensor pipe; its stage's scores are free then
            moves.append((scores + 1, pv, said, step))
        if pv < said and scores >= min(pv + 2, total):
            moves.append((scores, pv + 1, said, step))
        if said < total:
            if said < scores:
                moves.append((scores, pv, said + 1, step))
        elif wait == "o_full twice":
            if step == 0 and (n == 1 or passes(o_full(pv), n & 1)):
                moves.append((scores, pv, said, 1))
            if step == 1 and passes(o_full(pv), (n - 1) & 1):
                assert pv == total
                return False
        else:
            g = total - 1
            if passes(v_empty(pv, g & 1), (g >> 1) & 1):
                assert pv == total, "passed before the unit's last P V"
                return False
        return not moves or any(stuck(*m) for m in moves)

    if wait == "o_full twice" and n > 1:
        assert stuck(0, 0, 0, 0)
    else:
        assert not stuck(0, 0, 0, 0)


@pytest.mark.parametrize("verdict", ["a warp's", "the CTA's"])
@pytest.mark.parametrize("came", [(True, True), (True, False), (False, True), (False, False)])
def test_records_of_a_decode_cluster_that_come_late(verdict, came):
    """sdpa_decode_kernel, CLUSTER: two warps of a CTA have waited for the other CTAs' records, each by its own clock.  A warp that
    goes without them takes the cluster's barrier, which takes all threads that have not left; one that goes on takes the
    CTA's.  (Decided by each warp for itself, the two wait for one another for good.)"""
    if verdict == "the CTA's":  # __syncthreads_and, and who goes without leaves behind the cluster's barrier
        ways = [["cta", "cta"] if all(came) else ["cta", "cluster"]] * 2
    else:
        ways = [["cta"] if c else ["cluster", "cta"] for c in came]
    ways = [list(w) for w in ways]
    while any(ways) and all(w and w[0] == ways[0][0] for w in ways):  # a barrier opens when all who have not left are there
        ways = [w[1:] for w in ways]
    assert (not any(ways)) == (verdict == "the CTA's" or len(set(came)) == 1)
