"""Model of the operand ring of csrc/oz.cu: the waits for copies in flight at the end of a block that gave up."""
import itertools


def waits_end(totals, nbuf, fill):
    """Ring of nbuf slots filled by three warps each, which stopped after `totals` steps: do the waits for the last
    copies of every slot end? fill: a warp arrives without a copy in the steps that others have copied and it has not."""
    most = max(totals)
    arrivals = [sum(1 for t in totals if step < (most if fill else t)) for step in range(most)]
    waited = [range(max(0, (most if fill else t) - nbuf), most if fill else t) for t in totals]
    return all(arrivals[step] == 3 for steps in waited for step in steps)


def test_copies_are_waited_for_when_one_warp_stops_early():
    for nbuf in (2, 3, 8):
        for totals in itertools.product(range(2 * nbuf + 2), repeat=3):
            if max(totals) - min(totals) > nbuf:
                continue  # a step is copied once its slot's last use is complete, for which all three have copied it
            assert waits_end(totals, nbuf, True)
            assert waits_end(totals, nbuf, False) == (len(set(totals)) == 1)
