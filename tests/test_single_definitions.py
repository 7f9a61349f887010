"""One definition per name across the translation units (emergence_b200/csrc):
a function template or constexpr function that two .cu files define differently
outside `static` and anonymous namespaces is one symbol to the linker, which may
keep either body; a type likewise."""
import os
import re
from collections import defaultdict

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "emergence_b200", "csrc")
UNITS = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _definitions(text):
    """Names defined at namespace scope (column 0) with external linkage."""
    text = re.sub(r"//[^\n]*", "", text)
    text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)
    # anonymous namespaces, to their closing brace at column 0
    text = re.sub(r"^namespace \{.*?^\}", "", text, flags=re.S | re.M)
    names = set(re.findall(r"^struct (\w+)[^;{]*\{", text, re.M))
    for m in re.finditer(r"^(?:template\s*<[^\n]*?>\s+)?([A-Za-z_][\w:<>*& ]*?)\b(\w+)\s*\(([^;{}]*)\)[^;{}()]*\{", text, re.M):
        head = text[m.start():m.start(2)]
        if "static" not in head.split() and not head.startswith(("#", "struct", "namespace")):
            names.add(m.group(2))
    return names


def test_no_unit_defines_a_name_of_another():
    where = defaultdict(list)
    for f in UNITS:
        with open(os.path.join(CSRC, f), encoding="utf-8") as fh:
            for name in _definitions(fh.read()):
                where[name].append(f)
    assert "plan_sweeps" in where and "sweep_launch_fast" in where  # the scan sees definitions
    assert {n: f for n, f in where.items() if len(f) > 1} == {}
