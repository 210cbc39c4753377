"""The bounds-checked build's sites against its sources: every site has a check, every hand-over list and packed node list
is written through one, and every unit with checks is read out."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "multiq_workbench_gb300" / "csrc"


def _sources():
    return {p.name: p.read_text() for p in CSRC.glob("*.cu")}


def test_every_site_is_checked_somewhere():
    head = (CSRC / "mq_check.h").read_text()
    sites = set(re.findall(r"(MQ_SITE_\w+) = \d+", head))
    used = set(re.findall(r"MQ_SITE_\w+", " ".join(_sources().values())))
    assert sites == used, sites ^ used


def test_lists_that_kernels_fill_are_written_through_a_check():
    stores = 0
    for name, text in _sources().items():
        for m in re.finditer(r"(?<!\.)\b(hand|to|list|list_out)\[([^;]*?)\] = ", text):
            if m[2].strip() in ("base + __popc(m & ((1u << lane) - 1u))",):   # the first list of a call: one slot per ion by its ballot
                continue
            stores += 1
            assert m[2].startswith("MQ_CHK("), (name, m[0])
    assert stores >= 5


def test_every_unit_with_checks_is_read_out():
    engine = (CSRC / "mq_engine.cpp").read_text()
    readers = engine[engine.index("readers[]"):].split("}", 1)[0]
    for name, text in _sources().items():
        if "MQ_CHK" in text:
            m = re.search(r"MQ_CHECK_READER\((\w+)\)", text)
            assert m and m[1] in readers, name
