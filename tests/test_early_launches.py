"""The rules that make the step's early launches (programmatic serialization)
sound, read from the kernel source: a kernel waits for the one before it before
it lets its own dependent start, and none that may be resident while the kernel
before it writes reads the step's arrays through the non-coherent path.  No run
can show a stale line that the hardware happens not to keep."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KERNELS = os.path.join(ROOT, "sph-erosion_gb300", "csrc", "sph_kernels.cu")


def functions(text):
    """Bodies of the device functions and kernels, by name."""
    text = re.sub(r"//[^\n]*", "", text)
    out = {}
    for m in re.finditer(r"__(?:device|global)__[^;{}()]*?(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\(", text):
        i = text.index(")", m.end())
        while text[m.end():i].count("(") >= text[m.end():i + 1].count(")"):
            i = text.index(")", i + 1)
        j = i + 1
        if text[j:].lstrip()[:1] != "{":
            continue
        j = k = text.index("{", j)
        depth = 0
        while True:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            if depth == 0:
                break
            k += 1
        out[m.group(1)] = out.get(m.group(1), "") + text[j:k]
    return out


def reached(fns, name, seen):
    if name in seen or name not in fns:
        return seen
    seen.add(name)
    for callee in set(re.findall(r"\b(\w+)\s*(?:<[^;(){}]*>)?\(", fns[name])):
        reached(fns, callee, seen)
    return seen


def test_early_kernels_wait_first_and_read_coherently():
    text = open(KERNELS).read()
    fns = functions(text)
    enter = fns["step_enter"]
    assert 0 < enter.index("griddepcontrol.wait") < enter.index("griddepcontrol.launch_dependents")
    early = set(re.findall(r"launch\([^;]*?\b(k_\w+)", text))
    assert len(early) >= 8, early
    for k in early:
        assert re.match(r"\{\s*step_enter\((?:a\.)?early\);", fns[k]), k
        for f in reached(fns, k, set()):
            body = fns[f].replace("__ldg(tab + S.tab_off", "")  # row numbers: only copies write them
            assert "__ldg(" not in body and ".nc." not in body, (k, f)
