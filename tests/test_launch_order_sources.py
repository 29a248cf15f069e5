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


REMOTE = ("mapa", "shared::cluster.v2.f32", "dsmem_copy(", "mbar_arrive_cluster(")
CLUSTER_WAIT = ("cluster_wait()", "cluster_sync()")


def without_lambdas(body):
    """The body with its named lambdas taken out, and the names of those that reach another CTA's shared memory."""
    remote = set()
    while True:
        m = re.search(r"auto (\w+) = \[&\]\([^)]*\) \{", body)
        if m is None:
            return body, remote
        depth, j = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(body[j], 0)
            j += 1
        if first(body[m.end():j], REMOTE) is not None:
            remote.add(m.group(1) + "(")
        body = body[:m.start()] + body[j:]


@pytest.mark.parametrize("fname", sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")))
def test_another_ctas_shared_memory_is_touched_behind_a_cluster_barrier(fname):
    """A CTA of a cluster may store to another's shared memory, or arrive on its barriers, only once that CTA is known to run: the first
    half of a cluster barrier before it, and a second barrier that keeps the memory alive until everything has arrived."""
    for name, body in kernels(fname).items():
        main, remote = without_lambdas(body)
        use = first(main, REMOTE + tuple(sorted(remote)))
        if use is None:
            continue
        wait = first(main, CLUSTER_WAIT)
        assert wait is not None and wait < use, name
        last_use = max(main.rindex(w) for w in REMOTE + tuple(sorted(remote)) if w in main)
        assert max(main.rindex(w) for w in CLUSTER_WAIT if w in main) > last_use, name
