"""Every code a kernel leaves when it gives up a wait has a text in rq_check, and every text a kernel that leaves its code (no GPU)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "recipe_dev_b200" / "csrc"


def test_codes_and_texts_agree():
    sources = {p.name: p.read_text() for p in list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh"))}
    raised = {int(n) for text in sources.values() for n in re.findall(r"atomicExch\((?:p\.)?error_flag, (\d+)\)", text)}
    table = sources["rq_api.cu"].split("wait_code_text(int code) {")[1].split("default:")[0]
    texts = dict((int(n), t) for n, t in re.findall(r'case (\d+): return "([^"]+)";', table))
    assert raised and raised == set(texts)
    assert len(set(texts.values())) == len(texts)
