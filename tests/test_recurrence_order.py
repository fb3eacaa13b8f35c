"""Barrier phases of the two recurrences and of the chunk-parallel backward, from their source (see wait_model.py).

A wait on an mbarrier names a phase by its parity.  It is a wait for that phase only if the phase before is over
when it begins and the phase behind it cannot be over before it has been passed, whatever the parts take: by program
order and by arrivals that lead to waits.  A wait that can be overtaken stops its launch for good.  Nothing is
run on a device: a lost wait is a race."""

import re

import pytest
import wait_model


@pytest.mark.parametrize("kernel, form", wait_model.CASES)
def test_every_wait_sees_its_own_phase(kernel, form):
    assert wait_model.skipped_or_early(getattr(wait_model, kernel)(**form)) == []


@pytest.mark.parametrize("kernel, line, found", [
    # the state copy does not wait for the product that reads the copy before
    ("forward", r"if \(!NO_O && it > 0\) WAIT\(SB_FREE, .*\n", (1, "VN_DONE", "skipped")),
    # nor the issuer of w for the prep group's read of P, which takes the same columns
    ("forward", r"if \(!NO_O && it >= 0 && it >= lead && !WAITU\(P_FREE, .*\n", (1, "W_READY", "skipped")),
    # the tile of A may be loaded over before it has been scaled
    ("reverse", r"WAIT\(EMPTYA0 \+ sj, .*\n", (2, "FULLA0", "skipped")),
])
def test_a_missing_wait_is_found(kernel, line, found):
    """the lines are taken out of the text that the model reads, nowhere else"""
    text = open(f"{wait_model.CSRC}/{'fwd_tc.cu' if kernel == 'forward' else 'bwd_dh_tc.cu'}").read()
    without, n = re.subn(line, "\n", text)
    assert n == 1
    assert found in wait_model.skipped_or_early(getattr(wait_model, kernel)(lead=0, text=without))
