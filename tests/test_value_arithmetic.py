"""Approximate divisions belong to the bounds of the step skipping, which carry margins for
them, and to nothing whose result a record or a sign comes from: the fast evaluators divide
as the reference does."""
import os
import re

from gpis_extend_gb300 import build

# functions of flights.cu that return a bound with its own margin
BOUNDS = {"oct_skip_count", "reach_1d"}


def functions(code):
    """(name, body) of the functions and member functions of a file."""
    for m in re.finditer(r"\b(\w+)\s*\([^;{}()]*(?:\([^()]*\)[^;{}()]*)*\)\s*(?:const\s*)?\{", code):
        depth, k = 1, m.end()
        while depth and k < len(code):
            depth += {"{": 1, "}": -1}.get(code[k], 0)
            k += 1
        if m.group(1) not in ("if", "for", "while", "switch"):
            yield m.group(1), code[m.end():k]


def test_approximate_division_only_in_bounds():
    with open(os.path.join(build.CSRC, "flights.cu")) as f:
        code = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)
    users = {name for name, body in functions(code) if re.search(r"__fdividef|__frcp_|__frsqrt_|use_fast_math", body)}
    assert users <= BOUNDS, users
    in_bounds = sum(body.count("__fdividef") for name, body in functions(code) if name in BOUNDS)
    assert in_bounds == code.count("__fdividef") > 0
