"""What the kernels' barriers order, as their sources state it (no GPU needed)."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "frisk_b200" / "csrc"


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
