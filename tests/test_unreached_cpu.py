"""No-GPU check of the kernels' source: every function and constant that csrc defines is used somewhere in it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "helios_glm53flash_b200", "csrc")
DEFINITION = re.compile(r"^(?:template <[^\n]*>\s*)?(?:static|inline|constexpr|__device__|__host__|__global__)\b([^;={}\"]*)\)\s*(?:const\s*)?\{", re.M)
BOUNDS = re.compile(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)")
CONSTANTS = re.compile(r"\bconstexpr\s+[\w:]+\s+((?:\w+\s*=[^;]+));")


def test_nothing_in_csrc_is_out_of_reach():
    text = ""
    for path in sorted(p for e in ("cu", "cuh", "cpp") for p in glob.glob(os.path.join(CSRC, "*." + e))):
        t = re.sub(r"/\*.*?\*/", "", open(path).read(), flags=re.S)
        text += re.sub(r"//[^\n]*", "", t) + "\n"
    names = {m.group(1) for m in (re.search(r"\b(\w+)\s*\(", BOUNDS.sub("", d.group(1))) for d in DEFINITION.finditer(text)) if m}
    for m in CONSTANTS.finditer(text):
        names |= set(re.findall(r"(?:^|,\s*)(\w+)\s*=(?!=)", m.group(1)))
    assert {"prep_unit", "pdl_wait", "mla_pair_tc_kernel", "TKC_PIECES"} <= names      # the reader sees what there is
    assert sorted(n for n in names if len(re.findall(r"\b%s\b" % n, text)) < 2) == []
