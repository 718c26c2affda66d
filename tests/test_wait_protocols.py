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
