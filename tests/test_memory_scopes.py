"""Shared words that several blocks of a cluster update at once: PTX guarantees
the atomicity of two accesses only where the scope of each includes the other's
thread, and no run can show that it is missing -- so the source is read."""
import re
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent.parent / "bf-new_b200" / "csrc" / "resident.cu"


@pytest.mark.parametrize("name", ["shared_load", "shared_min", "shared_or"])
def test_cluster_form_has_cluster_scope(name):
    body = re.search(rf"__forceinline__ \w+ {name}\(.*?\n}}\n", SOURCE.read_text(), re.S).group(0)
    cluster, block = re.search(r"if \(kCluster\) \{(.*)\} else \{(.*)\}", body, re.S).groups()
    access = re.compile(r"\b(?:ld|st|red|atom)\.[\w.:]+")
    found = access.findall(cluster)
    assert len(found) == 2  # own block, any block
    assert all(".relaxed.cluster." in x for x in found), found
    assert len(access.findall(block)) == 1 and ".relaxed.cta." in access.findall(block)[0]
