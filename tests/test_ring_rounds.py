"""Ring depths of the weight-only kernel in csrc/umma_gemm.cu, evaluated from its configuration: every raw weight stage and every
operand stage has to be used by the same transform groups in each round of its ring.  A group that takes a stage over from
another one can pass the wait for it a whole phase early, which shows as a wrong tile once in many launches, if at all."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm-scaler_b200", "csrc", "umma_gemm.cu")


def _config(tok):
    """The integer constants of UmmaCfg<tok>."""
    with open(SRC) as f:
        body = re.search(r"template <int TOK> struct UmmaCfg \{(.*?)\n\};", re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read()), re.S).group(1)
    cfg = {"TOK": tok}
    for name, expr in re.findall(r"static constexpr int (\w+) = ([^;]+);", body):
        expr = " ".join(expr.split()).replace("/", "//")
        while "?" in expr:                                   # innermost conditional without parentheses inside, or the whole expression
            m = re.search(r"\(([^()?]*)\?([^()?:]*):([^()?:]*)\)", expr)
            if m:
                expr = expr[:m.start()] + "(%s if %s else %s)" % (m.group(2), m.group(1), m.group(3)) + expr[m.end():]
            else:
                c, rest = expr.split("?", 1)
                depth, at = 0, None
                for i, ch in enumerate(rest):
                    depth += (ch in "(?") - (ch == ")")
                    if ch == ":":
                        if depth == 0:
                            at = i
                            break
                        depth -= 1
                expr = "(%s) if (%s) else (%s)" % (rest[:at], c, rest[at + 1:])
        cfg[name] = int(eval(expr, {}, cfg))
    return cfg


@pytest.mark.parametrize("tok", [16, 32, 64, 128, 256])
@pytest.mark.parametrize("chunks_per_raw_stage", [2, 4])     # FP8, INT4
def test_a_stage_stays_with_its_groups(tok, chunks_per_raw_stage):
    c = _config(tok)
    raw, operand = {}, {}
    for chunk in range(240):
        group = chunk % c["NG"]
        raw.setdefault(chunk // chunks_per_raw_stage, set()).add(group)
        operand.setdefault(chunk % c["S"], set()).add(group)
    assert all(len(g) == 1 for g in operand.values())
    for stage, groups in raw.items():
        assert groups == raw[stage % c["RS"]]
    assert c["SMEM"] <= 232448 // c["CTAS"]
