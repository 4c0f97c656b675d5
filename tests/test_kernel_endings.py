"""How the tcgen05 kernels end, read from their sources: the warp that issues a CTA's products waits, on a count of its own,
until the tensor core has done all of them.  A wait on the CTA's abort flag ends after one look once another
wait has given up; the CTA would then free its tensor memory, and end, under products that are still running.  (Making a wait give up on
a GPU to see that is no test to run on one.)"""

from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tokensprint_b200" / "csrc"


@pytest.mark.parametrize("source", ["moe_tcgen05.cu", "variants/attention_tcgen05.cu"])
def test_the_issuing_warp_waits_for_its_products_whatever_gave_up(source):
    text = re.sub(r"//[^\n]*", "", (CSRC / source).read_text())
    commits = [m.end() for m in re.finditer(r"umma_commit\(smem_u32\(&(?:c\.)?all_done\)\)", text)]
    assert commits
    for at in commits:
        behind = text[at : at + 400]
        own = re.search(r"int (\w+) = 0;\s*mbar_wait\(smem_u32\(&(?:c\.)?all_done\), 0, &(\w+)\)", behind)
        assert own and own.group(1) == own.group(2), behind
        assert "__global__" not in behind[: own.start()]
