"""The products read weights before they wait for the launch before them, which is sound only while no kernel that writes weights lets its
dependents start early (no GPU: read from the sources)."""
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "recipe_dev_b200" / "csrc"


def test_writers_of_weights_signal_nothing_early():
    for name in ("rq_layout.cu", "rq_requant.cu", "rq_quantize.cu", "rq_decode.cuh"):
        code = "\n".join(line.split("//")[0] for line in (CSRC / name).read_text().splitlines())
        assert "launch_dependents" not in code and "programmatic" not in code, name
        assert "__global__" in code or name.endswith(".cuh")
