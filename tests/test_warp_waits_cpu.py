"""What the kernels' barriers order and what follows their bounded waits, as their sources state it (no GPU needed)."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "frisk_b200" / "csrc"
KERNELS = sorted(p.name for p in CSRC.glob("*.cu") if "mbar_wait" in p.read_text())


class Block:
    """A braced block of a source: what stands before its brace, and its statements without those of the blocks in it."""

    def __init__(self, head, outer):
        self.head, self.outer, self.own = head, outer, ""

    def one_lane(self):
        return bool(re.search(r"\b(lane|threadIdx\.x) == 0\b|elect_one\(\)", self.head)) or (self.outer is not None and self.outer.one_lane())


def places(name, pattern):
    """(block, place in its own statements) of every match of the pattern in a kernel's source."""
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    block, head, found = Block("", None), "", []
    for token in re.split(r"([{};])", text):
        if token == "{":
            block.own += head + "{}"
            block, head = Block(head, block), ""
        elif token == "}":
            block.own += head
            block, head = block.outer, ""
        else:
            found += [(block, len(block.own) + len(head) + m.start()) for m in re.finditer(pattern, token)]
            head += token
            if token == ";":
                block.own += head
                head = ""
    assert block.outer is None, name
    return found


def test_no_lane_reads_an_item_after_the_warp_has_released_it():
    """Attention: the producer writes a slot again when every consumer warp has arrived once, so the arrival comes after all lanes' reads."""
    reads = places("attention_fwd.cu", r"= item_slot\[")
    assert reads
    for block, at in reads:
        release = block.own.find("mbar_arrive(&item_empty", at)
        assert release >= 0 and (block.one_lane() or "__syncwarp()" in block.own[at:release])


@pytest.mark.parametrize("name", KERNELS)
def test_waits_of_whole_warps_are_voted_on(name):
    """A wait may run out for some lanes only, and votes, tensor-memory loads and __syncwarp need all of them.  So a per-lane wait belongs
    to code of one lane, or to a vote, or its outcome is voted on in the same block before anything else needs the warp, or it goes to a
    variable that nothing but votes reads."""
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    for block, at in places(name, r"\bmbar_wait(_both)?\("):
        before, after = block.own[:at], block.own[at:]
        if block.one_lane() or before.endswith("__all_sync(0xffffffffu, ") or re.search(r"lane == 0 && $", before):
            continue
        kept = re.search(r"(\w+) (&=|=) $", before)
        if kept and kept[1] != "ok":
            uses = re.findall(rf"(?:bool |__a(?:ny|ll)_sync\(0xffffffffu, !?)?\b{kept[1]}\b(?: &?= )?", text)
            assert all(re.match(r"bool |__a", use) or use.endswith("= ") for use in uses), (name, uses)
            continue
        vote = after.find("ok = __all_sync(0xffffffffu, ok)")
        assert vote >= 0 and not re.search(r"\{\}|break|return|_sync\(|__syncwarp|tmem_|elect_one", after[:vote]), (name, after[:80])


ALIGNED = r"\b(?:tmem_(?:ld|st)_32x32b_x\d+|tmem_st_wait|tmem_alloc(?:_pair)?|cluster_sync_all|load_scores|values|la\.store)\("
MEET = r"__sync(?:warp|threads)\(|_sync\(|\b(?:mbar_wait_warp|epi_sync|meet|combine_rows|cluster_sync_all|may_issue|issue_part|scores_there)\("
APART = r"if \([^;{}]*\b(?:lane|row|grow|threadIdx\.x) [<>=!]=?|if \(valid\)|clock64|\b[abl]+\.fetch\(|\bnote\("


def meets(text):
    """Where in a piece of source the warp meets, whichever way it goes (a block that begins and ends in the piece may be left out)."""
    opened, closed = [], []
    for i, c in enumerate(text):
        if c == "{":
            opened.append(i)
        elif c == "}" and opened:
            closed.append((opened.pop(), i))
    return [m.end() for m in re.finditer(MEET, text) if not any(a < m.start() < b for a, b in closed)]


@pytest.mark.parametrize("name", KERNELS)
def test_warps_meet_before_what_needs_all_lanes(name):
    """Instructions that a warp executes as one (tcgen05 loads, stores, waits and allocations, cluster barriers) come after a meeting of its
    lanes wherever code of single lanes comes before, in program order or in the loop's last round."""
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    opened, blocks = [], []
    for i, c in enumerate(text):
        if c == "{":
            opened.append(i)
        elif c == "}":
            blocks.append((opened.pop(), i))
    for m in re.finditer(ALIGNED, text):
        for begin, end in sorted((b for b in blocks if b[0] < m.start() < b[1]), reverse=True):  # from the innermost block outwards
            head = text[text.rfind("\n", 0, begin):begin]
            if re.search(r"warp == (?!0)", head) and m.group().startswith("tmem_alloc"):
                break  # (thread 0's set-up is another warp's)
            before = text[begin:m.start()]
            met = meets(before)
            piece = before[met[-1]:] if met else before
            if not met and re.search(r"\b(for|while) \(", head):
                rest = text[m.start():end]
                met_later = meets(rest)
                piece = (rest[met_later[-1]:] if met_later else rest) + piece
            apart = re.search(APART, piece)
            assert not apart, (name, text.count("\n", 0, m.start()) + 1, m.group(), apart.group())
            if met or re.search(r"__device__|\[&\]\(|\[\]\(|__launch_bounds__", head):
                break  # (a function is judged where it is called)
