"""Rules that the kernels' pipelines keep and that no run can show reliably, checked in
the sources."""
import os
import re

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "pynear_gb300", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return re.sub(r"//[^\n]*", "", text)


def _body(text, kernel):
    """The definition of a kernel, from its name to its closing brace."""
    at = re.search(r"\b%s\(const __grid_constant__" % kernel, text).start()
    i = text.index("{", at)
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
    raise AssertionError(kernel)


def test_slots_read_by_ordinary_loads_are_released_behind_a_proxy_fence():
    """A slot that copies refill and that a warp reads with ordinary loads: the release
    has to order those loads before the copies' writes (mbar_release_warp)."""
    scan = _body(_source("flat_scan.cu"), "float_scan_kernel")
    assert "mbar_release_warp(empty + slot)" in scan and "mbar_arrive(" not in scan
    topk = _body(_source("tc_scan.cu"), "tc_topk_kernel")
    assert "mbar_release_warp(nempty + ns)" in topk and "mbar_arrive(nempty" not in topk


def _waits_outside_one_thread(body):
    """mbar_wait calls in code that a whole warp runs and whose results may differ
    between its lanes."""
    found, scopes, i = [], [], 0
    head = ""  # text since the last brace or semicolon: what a block opens with
    for m in re.finditer(r"[{};]|\bmbar_wait\(", body):
        head += body[i:m.start()]
        i = m.end()
        if m.group() == "{":
            scopes.append(head)
            head = ""
        elif m.group() == "}":
            scopes.pop()
            head = ""
        elif m.group() == ";":
            head = ""
        else:
            one = any(re.search(r"if \(.*(lane|threadIdx\.x) == 0\b", s) for s in scopes)
            if not one and "__all_sync(0xffffffffu" not in head:
                found.append(head.strip() + " mbar_wait")
            head += m.group()
    return found


def test_waits_of_a_warp_have_one_answer():
    for name, kernel in (("flat_scan.cu", "float_scan_kernel"), ("tc_scan.cu", "tc_topk_kernel"),
                         ("tc_ivf.cu", "tc_ivf_kernel")):
        assert not _waits_outside_one_thread(_body(_source(name), kernel)), kernel


def test_an_early_end_waits_for_the_copies_that_were_issued():
    """The producer of a tensor-core scan whose wait ran out: what it waits for before
    the block ends is counted at the copies (a unit's or a tile's own count has moved on
    by then, and the other parity of a barrier is no wait at all)."""
    body = _body(_source("tc_scan.cu"), "tc_topk_kernel")
    at = body.index("auto settle")
    ends = re.findall(r"settle\(([^;]*)\);", body[at:])
    assert len(ends) == 3 and "(aloads - 1) & 1" in ends[2]
    issue = body[:at]
    assert re.search(r"&tmA[^;]*afull\);\s*\+\+aloads;", issue)
    assert re.search(r"bulk_load\(sscale[^;]*;\s*\+\+nloads;", issue)
    assert issue.count("++aloads") == 1 and issue.count("++nloads") == 1
    assert "nloads" in ends[1] or "x < nloads" in body[at:]
