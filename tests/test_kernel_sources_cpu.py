"""Source checks of what keeps programmatic dependent launches ordered (no
GPU): a kernel launched as a dependent waits for the kernel before it, and the
inline loads that such kernels use cannot be moved ahead of the wait.

A non-volatile asm is a function of its operands to the compiler, so a load
written as one may move above griddepcontrol.wait although that has a memory
clobber; a volatile one with a memory clobber may not."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "copss-hydrodynamics-private_gb300" / "csrc"
FREE = {"ld_piece"}  # loads of data that no kernel of a launch chain writes


def _sources():
    return {p.name: re.sub(r"//[^\n]*", "", p.read_text())
            for p in sorted(CSRC.iterdir()) if p.suffix in (".cu", ".cuh")}


def _closing(text, start):
    depth = 0
    for k in range(start, len(text)):
        depth += text[k] == "("
        depth -= text[k] == ")"
        if depth == 0:
            return k
    raise AssertionError("unbalanced")


def _enclosing(text, at):
    heads = [m for m in re.finditer(r"(\w+)\s*\([^;{}]*\)\s*\{", text[:at])
             if m.group(1) not in ("if", "for", "while", "switch")]
    return heads[-1].group(1)


def test_inline_loads_stay_behind_the_wait():
    seen = 0
    for name, text in _sources().items():
        for m in re.finditer(r"\basm\b(\s+volatile)?\s*\(", text):
            body = text[m.end() - 1:_closing(text, m.end() - 1)]
            if not re.search(r"\bld\.(global|relaxed|acquire|weak)", body):
                continue
            seen += 1
            if _enclosing(text, m.start()) in FREE:
                continue
            assert m.group(1) and '"memory"' in body, (name, body)
    assert seen >= 3
    # the free one reads the tensor's pieces only
    pair = _sources()["ggem_pair.cu"]
    uses = re.findall(r"ld_piece\(([^)]*)\)", pair)
    assert uses and all(u.startswith("const double4_32a *p") or u in ("r", "r + 1", "r + 2")
                        for u in uses)
    assert re.search(r"r = T\.rec \+ 3 \* idx;[^;]*ld_piece\(r \+ 2\)", pair)


def test_dependent_kernels_wait_for_the_one_before():
    sources = _sources()
    launched = set()
    for text in sources.values():
        for m in re.finditer(r"\blaunch_dependent(?:_cluster)?\s*\(", text):
            args = text[m.end():_closing(text, m.end() - 1)]
            head = args.split("dim3", 1)[0]  # the kernel, or a choice of kernels
            launched |= set(re.findall(r"\bk_\w+", head))
    assert len(launched) >= 20
    for k in sorted(launched):
        found = 0
        for text in sources.values():
            for m in re.finditer(r"__global__[^;{]*?\b" + k + r"\s*\(", text):
                body = text[text.index("{", _closing(text, m.end() - 1)):]
                depth, end = 0, 0
                for end, ch in enumerate(body):
                    depth += ch == "{"
                    depth -= ch == "}"
                    if depth == 0:
                        break
                assert "wait_prior_grid()" in body[:end], k
                found += 1
        assert found == 1, k
