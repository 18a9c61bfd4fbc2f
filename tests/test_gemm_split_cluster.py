"""What the clusters of gemm_split_sm100.cu owe each other, read from the kernel's source: a
cluster whose waits run out cannot be brought about on a GPU without risking a fault."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def kernel_body():
    with open(os.path.join(ROOT, "ptx.jl_b200", "csrc", "gemm_split_sm100.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    start = text.index("gemm_split_kernel(")
    return text[start:text.index("\n}\n", start)]


def test_no_cta_leaves_before_its_peers_stop_storing_into_it():
    """A CTA leaves when it has received everything its peers send it; if one of its waits ran
    out (its abort flag is up), only behind a cluster barrier that every peer reaches or leaves
    behind its last store, and behind the landing of the stores, which are asynchronous."""
    body = kernel_body()
    at = lambda token: [m.start() for m in re.finditer(re.escape(token), body)]
    arrive, wait, store = at("cluster_arrive()"), at("cluster_wait()"), at("st_async_v4(")
    assert len(arrive) == 2 and len(wait) == 2 and len(store) == 1
    assert arrive[0] < wait[0] < store[0] < at("mbar_wait<true>(bar_parts")[0] < arrive[1] < wait[1]
    assert wait[1] > max(at("__syncthreads()")[-1], at("tmem_dealloc(")[-1], at("store_acc_chunk16")[-1])
    closing = body[at("__syncthreads()")[-1]:]
    assert re.search(r"if \((kSplit|split > 1) && !misaligned && \*abort_flag != 0\) \{\s*cluster_arrive\(\);\s*cluster_wait\(\);", closing)
    assert at("mbar_try_wait(bar_parts")[0] > wait[1]
    assert "return" not in body          # no way past the closing wait


def test_the_wait_for_the_parts_acquires_at_cluster_scope():
    """Other CTAs store the parts, so a wait of this CTA's scope (the default) orders nothing."""
    assert "mbar_wait<true>(bar_parts" in kernel_body()
    with open(os.path.join(ROOT, "ptx.jl_b200", "csrc", "sm100_prims.cuh")) as f:
        prims = f.read()
    wait = prims[prims.index("bool mbar_try_wait("):]
    wait = wait[:wait.index("return ok")]
    assert "if constexpr (kCluster)" in wait and "mbarrier.try_wait.parity.acquire.cluster.shared::cta" in wait
    for caller in ("bool mbar_wait_slow(", "bool mbar_wait("):
        body = prims[prims.index(caller):]
        body = body[:body.index("\n}\n")]
        assert "mbar_try_wait<kCluster>" in body and "mbar_try_wait(" not in body
