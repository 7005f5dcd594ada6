"""The library's version number against what it stands for: the exported functions' arguments and the structs that callers fill."""
import hashlib
import os
import re

from lightllm_b200.csrc import build, ops

# the number -> what callers of that number were built for (see :func:`interface`).  Changed arguments or structs take the next number
# in csrc/common.cu, csrc/ops.py and csrc/host/generate.cpp, and a line here.
KNOWN = {25: "5eeac51547ca62c7", 26: "2619e82c8415ad5b"}


def interface() -> str:
    """A digest of the exported functions (result, name, types of the arguments in their order) and of the C structs of the headers."""
    found = []
    for name in sorted(os.listdir(build.CSRC_DIR)):
        if not name.endswith((".cu", ".h")):
            continue
        with open(os.path.join(build.CSRC_DIR, name)) as f:
            text = re.sub(r"/\*.*?\*/", " ", re.sub(r"//[^\n]*", " ", f.read()), flags=re.S)
        for ret, fn, args in re.findall(r"LLB_EXPORT\s+([\w\s\*]+?)\s*\b(llb_\w+)\s*\(([^)]*)\)\s*\{", text):
            types = [re.sub(r"\s*\w+$", "", " ".join(a.split())) for a in args.split(",")]
            found.append(" ".join(ret.split()) + " " + fn + "(" + ", ".join(types) + ")")
        if name.endswith(".h"):
            found += [" ".join(s.split()) for s in re.findall(r"typedef struct.*?\}\s*\w+\s*;", text, flags=re.S)]
    return hashlib.sha256("\n".join(sorted(found)).encode()).hexdigest()[:16]


def test_the_number_stands_for_this_interface():
    assert KNOWN.get(ops.ABI_VERSION) == interface(), f"callers built for {ops.ABI_VERSION} would misread this library: {interface()}"


def test_library_binding_and_program_agree():
    with open(os.path.join(build.CSRC_DIR, "host", "generate.cpp")) as f:
        program = int(re.search(r"EXPECTED_ABI = (\d+);", f.read()).group(1))
    assert program == ops.ABI_VERSION == ops.lib().llb_abi_version()
