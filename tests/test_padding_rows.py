"""Rows of a tile past the weight's last one cost no trips to memory in the product of bytes (no GPU: read from the source)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "recipe_dev_b200" / "csrc"


def test_scales_of_rows_that_are_not_there_are_not_copied():
    """Copied from the last row's place, past L1, they were one line of L2 that every CTA asked for at once."""
    scales = (CSRC / "rq_matmul_int8.cu").read_text().split("- the stored scales:")[1].split("cp.async.wait_all")[0]
    copies = re.findall(r"cp\.async\.cg\.shared\.global ([^;]*);\" ::(.*) : \"memory\"", scales)
    assert len(copies) == 1 and copies[0][0] == "[%0], [%1], 16, %2" and '"r"(row0 + i < p.rows ? 16 : 0)' in copies[0][1]
