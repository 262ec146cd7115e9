"""What a kernel that gave up a bounded wait is called in the report, against the codes in the kernels' sources."""

import pathlib
import re

from atomserve_b200.ops.status import describe

CSRC = pathlib.Path(__file__).resolve().parent.parent / "atomserve_b200" / "csrc"
FAMILIES = {  # sources that write the pipeline word, and what the report has to call them
    "gemm_tcgen05.cu": "GEMM:",
    "gemm_tcgen05_pair.cu": "GEMM on pairs",
    "attention_tcgen05.cu": "prefill attention",
    "attention_parts_tcgen05.cu": "prefill attention",
    "decode_chain.cu": "decode chain",
    "wait_selftest.cu": "self-test",
}


def _codes(text: str) -> set[int]:
    text = re.sub(r"//[^\n]*", "", text)
    for name, value in re.findall(r"constexpr int (k\w*Code) = (\d+);", text):
        text = text.replace(name, value)
    found = set()
    for last in re.findall(r"\b(?:mbar_wait|wait_or_give_up)\([^;]*?status, ([^;]*?)\)(?:;| \?| \&\&|\))", text):
        found.update(int(n) for n in re.findall(r"\b\d+\b", last.split(",")[0]))
    found.update(int(n) for n in re.findall(r"atomicExch\([^;]*status, (\d+)\)", text))
    return found


def test_every_wait_code_names_its_kernel():
    families = {}
    for name, family in FAMILIES.items():
        codes = _codes((CSRC / name).read_text())
        assert codes, f"no wait codes found in {name}"
        for code in codes:
            families.setdefault(code, set()).add(family)
    assert {code: names for code, names in families.items() if len(names) > 1} == {}
    for code, (family,) in families.items():
        assert family in describe([code, 0]), (code, describe([code, 0]))


def test_every_source_that_waits_is_listed():
    waiting = {p.name for p in CSRC.glob("*.cu") if re.search(r"\b(mbar_wait|wait_or_give_up)\(", p.read_text())}
    assert waiting <= set(FAMILIES)
