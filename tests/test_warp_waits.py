"""Waits of warps in which one lane acts on what all of them waited for (no GPU: read from the sources)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "recipe_dev_b200" / "csrc"


def test_the_streaming_producer_waits_by_vote():
    """A lane that looked late could meet the slot's next phase, and lanes that gave up alone would part from the others before a __syncwarp."""
    text = (CSRC / "rq_gemv_stream.cuh").read_text()
    assert "return __all_sync(0xffffffffu, mbar_wait(bar, parity, limit_ns));" in text.split("bool mbar_wait_warp(")[1].split("}")[0]
    producer = text.split("- producer warp")[1].split("- consumers")[0]
    assert "leader" in producer and len(re.findall(r"\bmbar_wait_warp\(", producer)) == 4
    assert not re.search(r"\bmbar_(try_)?wait\(", producer)
