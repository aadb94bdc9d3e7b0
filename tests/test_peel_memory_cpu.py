"""Rules of the peel's cross-block memory traffic, read from its source.

Blocks of a team hand data to one another under the GPU's memory model, whose
ordering only holds between accesses of the same width to the same word.  A
breach shows in no output of the hardware at hand, so the source is checked.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "kilosort_b200", "csrc")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def body(text, name):
    """Text of the definition of function `name`, from its name to its last brace."""
    start = re.search(r"\b%s\s*\([^;{]*\)\s*{" % re.escape(name), text)
    assert start, name
    depth, i = 1, start.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
    return text[start.start():i]


def test_barrier_accesses_have_one_width():
    common = source("ks_common.cuh")
    names = re.findall(r"\b(ks_grid_sync|ks_ctl_\w+)\s*\([^;{]*\)\s*{", common)
    assert "ks_grid_sync" in names
    widths = set()
    for n in names:
        text = body(common, n)
        widths |= {int(w) for w in re.findall(r'"(?:ld|st|red|atom)\.[\w.]*?\.[bus](\d+) ', text)}
        # the C++ atomics take their width from the word's type
        assert not re.search(r"reinterpret_cast<|\((?:unsigned|int)\s*\*\)", text), n
        if re.search(r"\batomic\w+\(", text):
            assert re.search(r"unsigned long long\s*\*\s*ctl", text), n
    assert widths == {64}
    # and the peel keeps no narrower pointer to the word
    assert not re.search(r"reinterpret_cast<(?:unsigned|int)\s*\*>\(team\)", source("peel_core.cuh"))


def test_pairs_keep_their_touch_list_to_themselves():
    """The warps that update a block's (block, group) pairs side by side have
    equal lists; none may store its own where another reads."""
    peel = source("peel_core.cuh")
    shared = [n for n in re.findall(r"\b(\w+)\s*\([^;{}()]*\)\s*{", peel)
              if "a.blist" in body(peel, n) and "reinterpret_cast<int*>(team" not in body(peel, n)]
    assert sorted(set(shared)) == ["group_scan", "unit_fetch"]
    # and a pair's inputs leave the published list out
    assert re.search(r"if \(kKind == kListed \|\| lane >= 8\) cp_async16", body(peel, "unit_fetch"))
    assert "run_units<kPair>" in body(peel, "scan_and_update")


def test_scratch_is_reused_behind_a_barrier():
    """A team's next batch overwrites the counts on which slower blocks leave the
    last one: a barrier lies between the loop's exits and the return."""
    peel = source("peel_core.cuh")
    run = body(peel, "run_peel")
    loop = run.index("++it) {")
    depth, i = 1, loop + len("++it) {")
    while depth:
        depth += {"{": 1, "}": -1}.get(run[i], 0)
        i += 1
    tail = run[i:]
    assert re.search(r"if \(again\b[^;]*ks_grid_sync\(a\.ctl", tail)
    multi = body(source("batched.cu"), "peel_multi_kernel")
    assert re.search(r"epoch,\s*i \+ n_teams < p\.n_batches\)", multi)
