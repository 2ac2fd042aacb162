"""Order within kernels that a run cannot show, read from their sources: what must lie ahead of griddep_wait_then_launch, and what behind it."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "crusaderbackend_b200", "csrc")


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def functions(text):
    """Bodies of a file's outermost functions (members of namespaces), comments taken out."""
    text = re.sub(r"//[^\n]*", "", text)
    for start in re.finditer(r"^[^\s#}/][^;{}]*\)\s*(?:const\s*)?\{$", text, re.M):
        end = text.find("\n}", start.end())
        yield text[start.start():end]


def allocates_in_order(body):
    """Every call of tmem_alloc, and a barrier of the whole block behind it, ahead of the first point from which a successor may start."""
    alloc, launch = body.rfind("tmem_alloc("), body.find("griddep_wait_then_launch(")
    return launch < 0 or 0 <= body.find("__syncthreads()", alloc) < launch


def test_columns_of_tmem_are_taken_before_a_successor_may_start():
    """A successor that starts first could take columns that another stream's kernel gives back, and wait for this kernel while it waits for them."""
    kernels = [(path, body) for path in sources() for body in functions(open(path).read()) if "tmem_alloc(" in body and "asm" not in body.split("{")[0] and "smem_u32" in body]
    assert len(kernels) >= 5
    wrong = [os.path.basename(path) for path, body in kernels if not allocates_in_order(body)]
    assert not wrong


@pytest.mark.parametrize("body, ok", [("{ tmem_alloc(a); __syncthreads(); griddep_wait_then_launch(); }", True), ("{ griddep_wait_then_launch(); tmem_alloc(a); __syncthreads(); }", False),
                                      ("{ __syncthreads(); if (copier) griddep_wait_then_launch(); else { tmem_alloc(a); griddep_wait_then_launch(); } }", False)])
def test_the_reader_sees_an_allocation_that_comes_late(body, ok):
    assert allocates_in_order(body) == ok


def movable_loads(text):
    """Inline loads from global memory that a compiler takes for functions of their operands, and may move ahead of a wait: those that are not
    volatile, nor read through a BehindWait, whose pointer depends on a volatile statement."""
    text, found = re.sub(r"//[^\n]*", "", text), []
    for m in re.finditer(r"\basm\s*\((?:[^;]|;(?=[^\n]*\"))*?\)\s*;", text):
        signature = re.findall(r"\n[^\s#}][^\n]*\)\s*\{", text[:m.start()])
        behind = bool(signature) and "(BehindWait src" in signature[-1] and '"l"(src.p' in m.group(0)
        if re.search(r"\bld\.(global|weak|relaxed|volatile)", m.group(0)) and not behind:
            found.append(m.group(0))
    return found


def test_loads_written_as_assembly_stay_behind_the_wait():
    wrong = {os.path.basename(path): movable_loads(open(path).read()) for path in sources()}
    assert not any(wrong.values()), wrong
    for path in sources():
        for body in functions(open(path).read()):
            if "const BehindWait " in body:  # made behind the wait itself
                assert 0 <= body.find("griddep_wait_then_launch(") < body.find("const BehindWait ")
    maker = open(os.path.join(CSRC, "gemm_simt.cu")).read()
    assert re.search(r"BehindWait\(const float\* q\) : p\(q\) \{ asm volatile\(\"\" : \"\+l\"\(p\)\); \}", maker)


def test_the_reader_sees_a_load_that_may_move():
    load = '\nfloat f(%s src, bool ok) {\n    asm%s("{ .reg .pred q; setp.ne.b32 q, %%2, 0;"\n        "@q ld.global.nc.f32 %%0, [%%1]; }" : "=f"(v) : "l"(%s), "r"(ok));\n    return v;\n}'
    assert len(movable_loads(load % ("const float*", "", "src"))) == 1 and not movable_loads(load % ("const float*", " volatile", "src"))
    assert not movable_loads(load % ("BehindWait", "", "src.p")) and len(movable_loads(load % ("BehindWait", "", "other"))) == 1
    assert not movable_loads('asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));')
