"""Source rules of the kernels that may start before their predecessor ends (those
that call pdl_wait): their data is read by plain loads (no __restrict__, no
__ldg but of context tables), since a read-only load may be moved above the wait,
and the kernel that takes tensor memory lets its successor start only then: no CTA
that a holder of columns waits for is still waiting for some itself."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pyfideslib_b200", "csrc")
FILES = ["ks.cu", "conv_tc.cu", "ntt_kernels.cuh"]


def _source(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def _kernels(src):
    """(kernel name, start, end) of every kernel, from __global__ to its closing brace."""
    for m in re.finditer(r"__global__", src):
        depth, i = 0, src.index("{", m.start())
        for j in range(i, len(src)):
            depth += {"{": 1, "}": -1}.get(src[j], 0)
            if depth == 0:
                break
        yield re.search(r"\b(k_\w+)\s*\(", src[m.start():j]).group(1), m.start(), j + 1


@pytest.mark.parametrize("name", FILES)
def test_early_kernels_wait(name):
    src = _source(name)
    launched = set(re.findall(r"launch(?:_pdl)?(?:<\w+>)?\(\s*(k_\w+)", src))
    waiting = {k for k, a, b in _kernels(src) if src[a:b].count("pdl_wait();") == 1}
    assert launched and launched <= waiting, launched - waiting


@pytest.mark.parametrize("name", FILES)
def test_data_is_read_by_plain_loads(name):
    src = _source(name)
    for k, a, b in reversed(list(_kernels(src))):  # kernels launched the ordinary way are free
        if "pdl_wait();" not in src[a:b]:
            src = src[:a] + src[b:]
    assert "__restrict__" not in src
    # context tables: by name, the twiddle and scale rows taken from them, and
    # conv_tc's byte matrix
    tables = ("ctx.", "twg,", "se,")
    if name == "conv_tc.cu":
        assert re.search(r"uint4\* src = reinterpret_cast<const uint4\*>\(\s*ctx\.tc_btab", src)
        tables += ("src + i)",)
    if name == "ntt_kernels.cuh":
        assert len(re.findall(r"uint64_t\* twg = \(fp \? ctx\.", src)) == 3
        src = src.replace("__ldg(reinterpret_cast<const ulonglong2*>(base) + idx)", "")  # ldg2 itself
        src = src.replace("ulonglong2 ldg2(const uint64_t* base, size_t idx)", "")
    for m in re.finditer(r"\b(__ldg|ldg2)\(", src):
        arg = re.sub(r"^reinterpret_cast<[^>]*>\(", "", src[m.end():m.end() + 80])
        assert arg.startswith(tables), arg


def test_successors_start_after_tensor_memory_is_taken():
    src = _source("conv_tc.cu")
    assert src.count("tcgen05.alloc") == 1 and src.count("pdl_trigger();") == 1
    (body,) = [src[a:b] for k, a, b in _kernels(src) if k == "k_conv_tc"]
    alloc, trigger = body.index("tcgen05.alloc"), body.index("pdl_trigger();")
    assert alloc < body.index("__syncthreads();", alloc) < trigger
    # every CTA that allocates also frees
    assert "return;" not in body[alloc:] and body.count("tcgen05.dealloc") == 1
