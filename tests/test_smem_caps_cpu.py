"""A kernel's shared-memory cap (cudaFuncSetAttribute) is one value for the whole process:
a cap that depends on a call's sizes can be lowered by another thread between setting and
launching.  Every cap in the sources is therefore a constant, named or written out."""
import glob
import os
import re

from conftest import PKG_DIR

CALL = re.compile(r"cudaFuncSetAttribute\(")
CONSTANT = re.compile(r"constexpr\s+(?:int|size_t|unsigned)\s+(\w+)\s*=\s*([^;]+);")


def _arguments(text, at):
    """The arguments of the call whose parenthesis opens before `at`."""
    depth, args, cur = 1, [], ""
    while depth:
        ch = text[at]
        depth += (ch == "(") - (ch == ")")
        if ch == "," and depth == 1:
            args.append(cur)
            cur = ""
        elif depth:
            cur += ch
        at += 1
    return [a.strip() for a in args + [cur]]


def test_caps_are_constants():
    found = 0
    for path in sorted(glob.glob(os.path.join(PKG_DIR, "csrc", "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        # (v->minb: a property of the kernel itself, of the variant's table entry)
        names = {m.group(1) for m in CONSTANT.finditer(text)} | {"sizeof", "v", "minb"}
        for m in CALL.finditer(text):
            args = _arguments(text, m.end())
            if "MaxDynamicSharedMemorySize" not in args[1]:
                continue
            found += 1
            cap = re.sub(r"\((?:int|size_t)\)", "", args[2])
            used = set(re.findall(r"[A-Za-z_]\w*", cap)) - {"int", "size_t", "float", "float2", "unsigned", "long"}
            assert used <= names, f"{os.path.basename(path)}: {args[0]}: cap {args[2]} is not a constant"
    assert found > 15
