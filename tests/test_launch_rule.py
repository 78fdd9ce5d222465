"""CPU: the order of griddepcontrol.wait and .launch_dependents in every kernel of the sources.

A kernel that lets its successor start before it has itself waited gives away what the successor's early reads rely on:
that everything launched before its predecessor is complete.  Only a kernel that is always an ordinary launch (nothing
before it is running any more) may trigger without a wait."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rotor-rag_b200", "csrc")


def kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__[^;{]*?\b(\w+)\s*\((?=[^;{]*\)\s*\{)(?:[^()]|\([^()]*\))*\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            yield os.path.basename(path), re.findall(r"(\w+_kernel)\b", m.group(0))[-1], text[m.end():i], text


FOUND = list(kernels())


def test_the_kernels_are_found():
    names = {name for _, name, _, _ in FOUND}
    assert {"bitlinear_acc_kernel", "row_stage_kernel", "vec_stage_kernel", "fused_gemv_kernel", "attn_decode_stream_kernel",
            "attn_decode_cluster_kernel", "dequant_kernel", "quantize_rows_kernel", "dense_gemm_t5_kernel"} <= names
    assert len(FOUND) == sum(len(re.findall(r"__global__", re.sub(r"//[^\n]*", "", open(p).read())))
                             for p in glob.glob(os.path.join(CSRC, "*.cu")))


@pytest.mark.parametrize("file,name", [(f, n) for f, n, b, _ in FOUND if "pdl_trigger()" in b])
def test_trigger_follows_wait(file, name):
    body, text = next((b, t) for f, n, b, t in FOUND if (f, n) == (file, name))
    waits, triggers = ([m.start() for m in re.finditer(w, body)] for w in (r"pdl_wait\(\)", r"pdl_trigger\(\)"))
    if not waits:
        assert re.search(name + r"(<[^;()]*>)?<<<", text) and not re.search(r"cudaLaunchKernelEx\([^;]*\b" + name, text), name
    else:
        assert len(waits) >= len(triggers) and all(w < t for w, t in zip(waits, triggers)), name


#: What no kernel of a call writes: weights and their scales, norms, tables, biases.  (r, rope, cs: (cos, sin) pairs.)
CONSTANTS = {"p.embed", "p.norm", "p.norm0", "p.norm1", "p.pro_norm", "p.st.norm1", "a.st.norm", "s.norm", "norm", "w", "b", "p.rope", "rope", "r",
             "cs", "cs4", "p.slopes", "p.sinks", "r.bias", "p.y_scales", "wscale_vec"}


def read_only(text):
    """Arguments of the non-coherent loads of a piece of source: the pointer that each starts from."""
    for m in re.finditer(r"\b__ldg\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield re.sub(r"^[&(]+", "", re.sub(r"reinterpret_cast<[^<>]*>\s*\(", "", text[m.end():i - 1])).lstrip("(& ")


def pointer(argument):
    return re.match(r"[\w.]+", argument).group(0)


@pytest.mark.parametrize("file,name", [(f, n) for f, n, b, _ in FOUND if "pdl_wait()" in b])
def test_dependent_kernels_read_what_others_write_with_coherent_loads(file, name):
    """A dependent kernel starts before the one in front of it has ended, so what that one writes is not read-only for the
    kernel's life, which a non-coherent load (__ldg, or a const __restrict__ parameter) takes for granted: it could be moved over
    the wait."""
    path = os.path.join(CSRC, file)
    text = re.sub(r"//[^\n]*", "", open(path).read())
    body = next(b for f, n, b, _ in FOUND if (f, n) == (file, name))
    head = re.search(r"\b" + name + r"\s*\(((?:[^()]|\([^()]*\))*)\)\s*\{", text).group(1)
    assert not re.search(r"const[^,]*__restrict__", head), head
    assert {pointer(a) for a in read_only(body)} <= CONSTANTS, name


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cuh"))), ids=os.path.basename)
def test_shared_device_code_reads_only_constants_with_non_coherent_loads(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    assert {pointer(a) for a in read_only(text)} <= CONSTANTS | {"p"}   # (p: ldg4, whose calls are below)
    for m in re.finditer(r"\bldg4\(([\w.]+)", text):
        assert m.group(1) in CONSTANTS | {"const"}, m.group(0)


def test_arrivals_at_another_ctas_barrier_release_at_cluster_scope():
    """An arrival without a scope orders memory within one CTA only: what a CTA writes for the other one of a pair needs the release
    of the whole cluster, and the waits that count such arrivals the acquire."""
    found = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"asm volatile\(((?:[^()\"]|\"[^\"]*\"|\([^()]*\))*)\)", text):
            arrive = re.search(r"mbarrier\.arrive([.\w:]*)\.shared::cluster", m.group(1))
            if not arrive or "tcgen05.commit" in m.group(1):
                continue
            found += 1
            fence = re.search(r"fence\.release\.sync_restrict::shared::cta\.cluster;", m.group(1)[:arrive.start()])
            assert ".release.cluster" in arrive.group(1) or (fence and ".relaxed.cluster" in arrive.group(1)), m.group(1)
    assert found
    body = next(b for _, n, b, _ in FOUND if n == "gemm_pair_kernel")
    waits = re.findall(r"t5_wait(<true>)?\(smem_u32\(&(s_full|s_acce|s_accf)\[", body)
    assert {bar for _, bar in waits} == {"s_full", "s_acce", "s_accf"} and all(peer for peer, _ in waits)
