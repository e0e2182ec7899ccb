"""The rule of the chained kernels of the plasma slice loop (gem-pic-3d_b200/csrc/k_pdl.cuh), checked on their source: a kernel
that is launched as a programmatic dependent is resident while the kernel before it still writes, so what that one writes must
not be read as constant memory (`const __restrict__` parameters, __ldg), which the compiler may load non-coherently or ahead
of the wait. No run can show this: a build that happens to keep the order passes every comparison.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "gem-pic-3d_b200", "csrc")
# the chained kernels, and of each what the kernel directly before it writes: kernel parameters, and members of StreamArgs
CHAIN = {
    "k_stream": ([], ["Fmid", "F", "Fd"]),                  # after the rows of the real fields
    "k_ss_rows": (["J"], []),                               # after the push's deposit
    "k_pass_cols": (["T0", "T1", "T2"], []),                # after the rows of the current's spectra
    "k_rf_row_slice": (["W0", "W1", "W2", "W3", "W4", "W5"], []),   # after the columns
}


def sources():
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".hpp")):
            with open(os.path.join(CSRC, f)) as fh:
                out[f] = re.sub(r"//[^\n]*", "", fh.read())
    return out


def balanced(s, i, o, c):
    depth = 0
    for j in range(i, len(s)):
        depth += (s[j] == o) - (s[j] == c)
        if depth == 0:
            return s[i + 1:j], j
    raise ValueError("unbalanced")


def kernel(src, name):
    """Parameter list and body of a __global__ kernel."""
    for text in src.values():
        for m in re.finditer(r"\b" + name + r"\s*\(", text):
            head = text[max(0, m.start() - 300):m.start()]
            if "__global__" not in head[max(head.rfind(";"), head.rfind("}")) + 1:]:
                continue
            params, j = balanced(text, m.end() - 1, "(", ")")
            body, _ = balanced(text, text.index("{", j), "{", "}")
            return [re.sub(r"\s+", " ", p).strip() for p in params.split(",")], body
    raise AssertionError(f"{name}: no such kernel")


def test_every_chained_kernel_is_covered():
    src = sources()
    launched = set()
    for f, text in src.items():
        if f == "k_pdl.cuh":
            continue
        for m in re.finditer(r"launch_pdl\(", text):
            args, _ = balanced(text, m.end() - 1, "(", ")")
            k = args.split(",")[1].strip()
            k = re.match(r"\w+", k).group(0)
            if k == "kern":                               # the function pointer's value, set or passed nearby
                near = text[max(0, m.start() - 900):m.start()] + text[m.start():m.start() + 1200]
                names = set(re.findall(r"\b(k_\w+)<", near)) & set(CHAIN)
                assert names, (f, "launch_pdl of an unknown kernel")
                launched |= names
            else:
                launched.add(k)
    assert launched == set(CHAIN)


def test_handed_over_parameters_promise_nothing():
    src = sources()
    for name, (handed, _) in CHAIN.items():
        params, body = kernel(src, name)
        for h in handed:
            p = [q for q in params if re.search(r"\b" + h + "$", q)]
            assert len(p) == 1, (name, h)
            assert "__restrict__" not in p[0] and "const" not in p[0], (name, p[0])
            assert not re.search(r"__ldg\(&?\s*" + h + r"\b", body), (name, h)
        if name == "k_stream":
            continue
        wait = body.index("pdl_wait()")
        assert wait < body.index("pdl_next()"), name
        for h in handed:                                  # first used behind the wait
            assert not re.search(r"\b" + h + r"\b", body[:wait]), (name, h, "read before the wait")


def test_the_push_gathers_by_ordinary_loads():
    text = sources()["k_plasma.cu"]
    for h in os.listdir(CSRC):
        if h.startswith("k_stream"):
            text += sources()[h]
    seen = 0
    for m in re.finditer(r"\b(sgather\w*|field_abs\w*)\s*\(const StreamArgs& c", text):
        _, j = balanced(text, text.index("(", m.start()), "(", ")")
        body, _ = balanced(text, text.index("{", j), "{", "}")
        assert "__ldg" not in body and "__restrict__" not in body, m.group(1)
        seen += 1
    assert seen >= 5
    hpp = sources()["g3d_plasma.hpp"]
    args, _ = balanced(hpp, hpp.index("{", hpp.index("struct StreamArgs")), "{", "}")
    for m in CHAIN["k_stream"][1]:
        decl = [d for d in args.split(";") if re.search(r"\b" + m + r"$", d.strip())]
        assert len(decl) == 1 and "__restrict__" not in decl[0], m
