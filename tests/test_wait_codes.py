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


def test_a_code_of_the_integer_products_names_what_was_waited_for():
    """One code a barrier there, and its text speaks of it: scales are not activations, and what a copy lands nobody staged."""
    waits = re.findall(r"mbar_wait_warp\(&(\w+)\b[^;]*?atomicExch\(p\.error_flag, (\d+)\)", (CSRC / "rq_matmul_int8.cu").read_text())
    codes = {}
    for barrier, code in waits:
        codes.setdefault(barrier, set()).add(int(code))
    assert len(waits) == 13 and all(len(c) == 1 for c in codes.values()) and len(set.union(*codes.values())) == len(codes), codes
    texts = {int(n): t for n, t in re.findall(r'case (\d+): return "([^"]+)";', (CSRC / "rq_api.cu").read_text())}
    said = {"scales_full": "stored scales never arrived", "scales_free": "stored scales: a slot", "a_full": "copied as it is stored", "a_free": "operand slot", "b_full": "activations never arrived",
            "b_free": "activation copies: a slot", "done": "sum", "drained": "accumulator", "raw_full": "stored bytes never", "freed": "stored bytes: a slot", "ended": "products", "full": "copies"}
    assert set(said) == set(codes)
    for barrier, words in said.items():
        assert words in texts[min(codes[barrier])], barrier
