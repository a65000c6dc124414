"""Rules of the kernels' bounded waits that no run shows, because they matter once a wait is given up: read from the sources (no GPU needed)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cera_b200", "csrc")


def _sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        yield os.path.basename(path), re.sub(r"//[^\n]*", "", open(path).read())


# Waits that a thread makes for itself: it is alone, or meets no instruction that reads other lanes before they are together again.
BY_THREAD = {"attention_exact.cu": 1,  # the thread that requests V
             "attention_tc.cu": 2,     # the thread that requests operands
             "gemm_tc.cu": 2,          # weight producers, each with operands of its own
             "gemv_exact.cu": 3,       # lanes stay in step: none is missing from what follows
             "gemv_tma.cu": 1}         # the thread that requests rows


def test_a_warp_decides_together_whether_a_wait_was_given_up():
    alone = {}
    for name, text in _sources():
        for call in re.finditer(r"\bmbar_wait(_blocking)?\(", text):
            ahead = re.split(r"[;{}]", text[:call.start()])[-1]  # the statement's beginning
            if name == "tma.cuh" or ahead.rstrip().endswith("bool") or "__all_sync(" in ahead:
                continue
            alone[name] = alone.get(name, 0) + 1
    assert alone == BY_THREAD


def test_a_loader_that_gave_up_waits_for_its_copies():
    """Kernels with a warp that requests operands ahead: shared memory may not go to another CTA with a copy on its way into it."""
    asked = {}
    for name, text in _sources():
        for body in text.split("__global__")[1:]:
            if "tc_commit" in body and re.search(r"\b(bulk|tensor)_g2s\w*\(", body):
                asked[re.search(r"(\w+_kernel)\(", body).group(1)] = bool(re.search(r"abort_flag\).*mbar_test\(", body, re.S))
    assert len(asked) == 5 and all(asked.values()), asked


def test_a_plain_arrival_at_another_cta_hands_over_tmem_only():
    """Its scope is the CTA it comes from: what that CTA's copies or threads wrote to memory is not part of it."""
    seen = 0
    for name, text in _sources():
        for call in re.finditer(r"\bmbar_arrive_cluster\(tma::", text):
            seen += 1
            assert "tc_fence_before();" in text[:call.start()][-250:], name
    assert seen == 2


def test_every_barrier_of_a_loaders_copies_is_waited_for():
    """The wide prompt product has two: the stages' and the factors' (whose copies no stage's barrier counts)."""
    body = dict(_sources())["gemm_tc.cu"].split("gemm_tcw_kernel(const TcParams")[1].split("__global__")[0]
    drain = body[body.index("if (PAIR || *abort_flag)"):]
    assert re.search(r"mbar_test\(last \+", drain) and re.search(r"mbar_test\(full_v \+", drain)
