"""What the pair kernels and their callers share is declared once."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "rpeg_b200" / "csrc"


def test_pair_declarations_stand_in_one_header():
    texts = {p.name: p.read_text() for p in (*CSRC.glob("*.cu"), *CSRC.glob("*.cuh"), *CSRC.glob("*.h"))}
    assert [n for n, t in texts.items() if re.search(r"struct PairPlan\s*\{", t)] == ["pair.cuh"]
    for name in ("gemm_pair", "gemm_pair_swiglu", "pair_plan", "moe_pair"):
        declared = [n for n, t in texts.items() if re.search(r"^(?:int|PairPlan) %s\([^;{]*\);" % name, t, re.M)]
        assert declared == ["pair.cuh"], (name, declared)
