"""The rule of launch_next() (csrc/common.cuh), checked on the sources: a kernel that it
launches starts with begin_after_previous(), only copies of pointers before it, and
gives it every pointer whose loads the compiler may otherwise move up: __restrict__
parameters that the kernel reads, and pointers read through __ldg."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _sources():
    text = ""
    for p in sorted(glob.glob(os.path.join(ROOT, "gbm3d_b200", "csrc", "*.cu*"))):
        with open(p) as f:
            text += re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S) + "\n"
    return text


def _close(s, i, opening, closing):
    """Index after the bracket that closes the one at i."""
    depth = 0
    for k in range(i, len(s)):
        depth += (s[k] == opening) - (s[k] == closing)
        if depth == 0:
            return k + 1
    raise ValueError("unbalanced")


def _launched(src):
    names = set()
    for m in re.finditer(r"launch_next\(\s*(\w+)", src):
        if m.group(1).startswith("k_"):
            names.add(m.group(1))
        elif m.group(1) == "kern":  # chosen just before
            pick = src[src.rindex("auto kern =", 0, m.start()):]
            names.update(re.findall(r"\bk_\w+", pick[:pick.index(";")]))
    return names


def _kernel(src, name):
    m = re.search(r"__global__[^;{}]*?\b" + name + r"\(", src)
    end = _close(src, m.end() - 1, "(", ")")
    start = src.index("{", end)
    return src[m.end():end - 1], src[start + 1:_close(src, start, "{", "}") - 1]


def violations(params, body):
    out = []
    head, sep, rest = body.partition("begin_after_previous(")
    if not sep:
        return ["no begin_after_previous()"]
    given = set(re.findall(r"\w+", rest[:rest.index(")")]))
    for st in head.split(";")[:-1]:
        if not re.fullmatch(r"\s*const \w+\* \w+ = A\.\w+\s*", st):
            out.append("before begin_after_previous(): " + st.strip())
    copies = set(re.findall(r"(\w+) = A\.", head))
    for p in params.split(","):
        m = re.search(r"__restrict__ (\w+)", p)
        if not m:
            continue
        name = m.group(1)
        reads = p.strip().startswith("const")
        for a in re.finditer(r"\b" + name + r"\[", rest):  # else: an element that is not just assigned
            reads |= not re.match(r"\s*=[^=]", rest[_close(rest, a.end() - 1, "[", "]"):])
        if reads and name not in given:
            out.append(f"reads {name} without giving it")
    for name in re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?\s*(\w+)", rest):
        if name in copies and name not in given:
            out.append(f"__ldg of {name} without giving it")
        if re.search(r"\* " + name + r" = [^;]*\bA\.", rest):
            out.append(f"__ldg of {name}, taken from the arguments after the wait")
    return out


def test_kernels_of_launch_next_begin_after_the_previous_one():
    src = _sources()
    names = _launched(src)
    assert len(names) >= 15
    bad = {n: v for n in sorted(names) if (v := violations(*_kernel(src, n)))}
    assert not bad, bad


def test_the_check_sees_a_broken_rule():
    good = "begin_after_previous(v); out[0] = v[0];"
    assert not violations("const float* __restrict__ v, float* __restrict__ out", good)
    assert violations("const float* __restrict__ v, float* __restrict__ out", "out[0] = v[0];")
    assert violations("const float* __restrict__ v, float* __restrict__ out", good.replace("(v)", "()"))
    assert violations("const float* __restrict__ v, float* __restrict__ out", "int a = v[0]; " + good)
    assert violations("const float* __restrict__ v, float* __restrict__ out", good + " out[1] = out[2];")
    assert violations("Args A", "const float* p = A.p; begin_after_previous(); out[0] = __ldg(p + 1);")
    assert violations("Args A", "begin_after_previous(); const float* p = A.p; out[0] = __ldg(p + 1);")
