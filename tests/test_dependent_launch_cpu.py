"""Kernels that may start before the kernels ahead of them have ended: each waits before it reads, and reads with loads that the
wait orders (csrc/kernels/dependent_launch.h)."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parents[1] / "coccl_b200" / "csrc" / "kernels"
UNITS = sorted(p.name for p in KERNELS.glob("*.cu") if "dependent_launch.h" in p.read_text())


def _code(path):
    text = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def _headers(path, seen):
    for name in re.findall(r'#include "([^"]+)"', path.read_text()):
        header = KERNELS / name
        if header.exists() and header not in seen:
            seen.add(header)
            _headers(header, seen)
    return seen


def _functions(code):
    """(name, text) of the functions at the outermost level of a namespace."""
    starts = [m.start() for m in re.finditer(r"^(?:template\b[^\n]*\n)?(?:static |extern \"C\" )?(?:__global__|__device__|__host__|int|void|long|inline)\b",
                                             code, flags=re.M)]
    for a, b in zip(starts, [*starts[1:], len(code)]):
        body = code[a:b]
        name = re.search(r"(\w+)\s*\((?![^()]*\)\s*\w+\s*\()", re.sub(r"__launch_bounds__\([^)]*\)", "", body))
        yield (name.group(1) if name else ""), body


# read-only loads, and pointers that let the compiler make them
UNORDERED = re.compile(r"__ldg\s*\(|ld\.global\.nc|const\s+[\w:<>]+\s*\*\s*__restrict__")


def test_there_are_such_kernels():
    assert {"train_kernels.cu", "embed_kernels.cu", "llama_kernels.cu", "gemm_small_kernels.cu"} <= set(UNITS)


@pytest.mark.parametrize("unit", UNITS)
def test_no_read_only_loads(unit):
    source = _code(KERNELS / unit)
    assert not UNORDERED.findall(source)
    for header in _headers(KERNELS / unit, set()):
        code = _code(header)
        used = [(n, t) for n, t in _functions(code) if not n or n in source]
        rest = code   # structures with members (Vec8 and the like) count as a whole
        for n, t in _functions(code):
            if (n, t) not in used:
                rest = rest.replace(t, "")
        assert not UNORDERED.findall(rest), f"{header.name} reads with loads that the wait does not order"


@pytest.mark.parametrize("unit", UNITS)
def test_every_dependent_kernel_waits_first(unit):
    """Every kernel of these files that is launched as a dependent lets the next one start and waits for the one before, outside any
    branch, ahead of every access to its arguments' memory. The small GEMM sets itself up first and lets the next one start late."""
    source = _code(KERNELS / unit)
    launched = set(re.findall(r"launch(?:After\(|IfEarly\(\w+,)\s*(\w+)", source)) | set(re.findall(r"cudaLaunchKernelEx\([^,]+,\s*(\w+)", source))
    assert launched
    kernels = {n: t for n, t in _functions(source) if "__global__" in t}
    for name in launched:
        body = kernels[name]
        late = unit == "gemm_small_kernels.cu"
        waits = re.search(r"^  awaitPrevious\(\);" if late else r"^  releaseNext\(\);\n  awaitPrevious\(\);", body, flags=re.M)
        assert waits and re.search(r"^  releaseNext\(\);", body, flags=re.M), f"{name} does not wait"
        ahead = body[body.index("{", body.index(name)):waits.start()]
        assert late or not ahead.strip("{ \n"), f"{name} does something ahead of its wait"
