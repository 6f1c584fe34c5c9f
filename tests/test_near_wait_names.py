"""The names that the binding gives the wait counters of the tensor-core near field, against the waits in the engine's
source: every wait code has a name of the role that waits, and no name stands for a counter that nothing writes."""
import os
import re

from conftest import REPO
from hignn_b200 import capi


def test_names_follow_the_engine():
    with open(os.path.join(REPO, "hignn_b200", "csrc", "tc_mlp.cuh")) as fh:
        text = re.sub(r"//[^\n]*", "", fh.read())
    found = {}
    for role, prefix in (("MmaWarp", "mma_"), ("Epi", "epi_"), ("Server", "server_")):
        start = text.index(f"struct {role} ")
        body = text[start:text.index("\n};", start)]
        for code in re.findall(r"wait\([^;{]*?,\s*(\d\d)(?:,[^)]*)?\)", body):
            found[int(code) - 13] = prefix
    consts = {k: int(v) for k, v in re.findall(r"(kProfTotal|kProfTiles) = (\d+)", text)}
    names = dict(capi.NEAR_WAIT_SLOTS)
    assert names.pop(consts["kProfTotal"]).endswith("total_warp0") and names.pop(consts["kProfTiles"]) == "tiles"
    assert set(names) == set(found)
    for slot, prefix in found.items():
        assert names[slot].startswith(prefix)
