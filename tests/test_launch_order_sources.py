"""What a kernel may do ahead of its dependency wait, read from the sources: a mistake here is a race on a weight, which shows on a
GPU only now and then.

The GEMV kernels on quantised activations stream their weight before griddepcontrol.wait (the header says so).  A host that writes
a weight on the stream, quantises the activations and calls the GEMV relies on the quantiser between them: no kernel behind it may
start before everything in front of it has finished.  The single-row GEMV on f32 activations is not in the header's list of early
readers, so it reads nothing and lets nothing start ahead of its own wait."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tensorpencil_b200", "csrc")
WAIT = ("tpb_grid_dep_wait()", "griddepcontrol.wait")
TRIGGER = ("tpb_grid_dep_launch()", "griddepcontrol.launch_dependents")
EARLY_READERS = {"qgemv.cu": {"q8_0_gemv_q8n_kernel"}, "qgemv_mma.cu": {"q8_0_gemv_mma_kernel"},
                 "qgemv_k.cu": {"kquant_gemv_q8n_kernel", "kquant_gemv_ring_kernel", "q6k_gemv_q8n_kernel", "q6k_gemv_ring_kernel"},
                 "qgemv_kmma.cu": {"kquant_gemv_mma_kernel"}}


def kernels(fname):
    """name -> body of every __global__ function of a source file, comments removed."""
    with open(os.path.join(CSRC, fname)) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    out = {}
    for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\(", src):
        i = src.index("{", m.end())
        depth, j = 1, i + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(src[j], 0)
            j += 1
        out[m.group(1)] = src[i:j]
    return out


def first(body, words):
    at = [body.index(w) for w in words if w in body]
    return min(at) if at else None


@pytest.mark.parametrize("fname,name", [("qgemv.cu", "q8_1_quantize_kernel"), ("qgemv.cu", "q8_0_gemv_f32_ring_kernel")])
def test_nothing_behind_it_starts_before_its_wait(fname, name):
    body = kernels(fname)[name]
    wait, trigger = first(body, WAIT), first(body, TRIGGER)
    assert wait is not None
    assert trigger is None or wait < trigger


@pytest.mark.parametrize("fname", sorted(f for f in os.listdir(CSRC) if f.startswith("qgemv") and f.endswith(".cu")))
def test_only_the_listed_kernels_copy_before_their_wait(fname):
    found = kernels(fname)
    early = EARLY_READERS.get(fname, set())
    assert early <= set(found)
    for name, body in found.items():
        copy = first(body, ("bulk_g2s(", "cp.async.bulk"))
        if name in early or copy is None:
            continue
        wait = first(body, WAIT)
        assert wait is not None and wait < copy, name
