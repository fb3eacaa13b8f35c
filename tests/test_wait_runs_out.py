"""What a block does when one of its bounded waits runs out, from the kernels' source (see wait_model.py): each
wait of the first and the last warp of every role in turn; of the waits that are then left open, the ones of the
first or of the last warps run out first.  Nothing of that is run on a device; the last test times a wait that runs
out there."""

import os
import re

import pytest
import wait_model

FORMS = [("forward", dict(n_it=2)), ("forward", dict(n_it=2, lead=1, extra=True, partial=True)),
         ("forward", dict(n_it=2, no_o=True, extra=True)), ("forward", dict(n_it=2, no_o=True)),
         ("reverse", dict(n_it=2, partial=True)), ("items", dict(n_items=2, partial=(1,))),
         ("items", dict(n_items=2, clc=True))]


@pytest.fixture(scope="module", params=FORMS, ids=lambda f: "-".join([f[0], *f[1]]))
def plays(request):
    """the kernel, and of every play (warps left at a named barrier, what a warp signalled or issued behind its
    own wait)"""
    name, form = request.param
    kernel = getattr(wait_model, name)(**form)
    warps = (0, 7, 8, 15, 16) if name == "items" else [w for w in range(kernel.warps) if w < 4 or w % 4 in (0, 3)]
    return kernel, [wait_model.given_up(kernel, w, nth, bool(nth & 1)) for w in warps
                    for nth in range(wait_model.waits_of(kernel, w))]


def test_every_warp_comes_to_the_end(plays):
    assert [left for left, _ in plays[1] if left] == []


def test_no_gradient_of_an_incomplete_item_is_stored(plays):
    assert {(w, e) for _, late in plays[1] for w, e in late if e[1] in ("dv", "store_rows")} == set()


def test_nothing_is_issued_or_signalled_behind_a_wait_that_ran_out(plays):
    """...by the warp that waited: copies, products and arrivals may outlive the block or pass for the ones of
    complete work (SETTLED is the end of what it had issued before)"""
    kernel, results = plays
    assert {(w, e) for _, late in results for w, e in late if e[1] != kernel.names["SETTLED"]} == set()


@pytest.mark.parametrize("file", ["fwd_tc.cu", "bwd_dh_tc.cu", "prep_kernels.cu"])
def test_a_warp_goes_on_or_leaves_as_one(file):
    """Each lane counts its own tries, and what stands behind a wait are instructions of whole warps: a look at the
    count decides for the warp (a vote), for a group (a barrier's) or for what one lane does alone."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(wait_model.CSRC, file)).read())
    alone = (r"__all_sync\(0xffffffffu, tries > 0\)", r"bar_all<\d+, \d+>\(tries > 0\)", r"elect_one\(\) && tries > 0",
             r"if \(tries <= 0\) \*abort_flag = 1;", r"if \(tries <= 0\) atomicCAS\(", r"if \(tries > 0\) mbar_arrive\(",
             r"lane == 0 && tries > 0\) mbar_arrive\(", r"tries > 0 \?")
    looks = re.findall(r"[^\n]*\btries (?:>|<=) 0[^\n]*", text)
    assert looks
    assert [line.strip() for line in looks if not any(re.search(a, line) for a in alone)] == []


@pytest.mark.gpu
def test_a_wait_is_given_up_after_about_a_second():
    """WAIT_TRIES times what a try takes where nobody arrives"""
    import ctypes

    import torch

    from flashqla_b200 import _lib

    lib, stream = _lib.load(), torch.cuda.current_stream().cuda_stream
    tries = 1 << int(re.search(r"WAIT_TRIES = 1 << (\d+);", open(os.path.join(wait_model.CSRC, "tc05.cuh")).read())[1])
    took = []
    for n in (1, 50, 100):  # (the first launch loads the kernel)
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        begin.record()
        assert lib.fqla_selftest_wait_timeout(n, stream) == 0
        end.record()
        torch.cuda.synchronize()
        took.append(begin.elapsed_time(end))
    assert lib.fqla_device_status(ctypes.byref(ctypes.c_int()), 1) == 0
    assert 0.2 < (took[2] - took[1]) / 50 / 1000 * tries < 5
