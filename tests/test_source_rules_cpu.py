"""Rules of the kernel sources that no run can show broken without hanging a GPU, checked by reading."""
import os
import re

from conftest import ROOT


def test_warps_of_the_tensor_core_gemm_leave_a_wait_as_a_whole():
    """A bounded wait that gives up is seen by the lanes of a warp at different times.  Wherever a wait is followed by instructions
    of the whole warp (tcgen05.ld / st / wait, __syncwarp), its result has to be voted on first; only the TMA producer waits in a
    single lane."""
    src = open(os.path.join(ROOT, "tace_b200", "csrc", "tc_gemm.cu")).read()
    roles = re.split(r"// ---- (TMA producer|MMA issuer|operand splitters|epilogue)", src)[1:]
    bodies = dict(zip(roles[::2], roles[1::2]))
    assert len(bodies) == 4
    assert re.match(r"\s*if \(lane == 0\) \{", bodies["TMA producer"])
    for role in ("operand splitters", "epilogue"):
        body = bodies[role].split("tcgen05.dealloc")[0]
        assert "sync.aligned" in body or "tmem_" in body
        assert re.search(r"\bwarp_wait\(", body) and not re.search(r"\bmbar_wait\(", body), role
    issuer = bodies["MMA issuer"]
    last_wait = issuer.rindex("mbar_wait(")
    assert "__all_sync(" in issuer[last_wait:issuer.index("umma_tf32_ts(")]
    assert "__all_sync(" in src[src.index("bool warp_wait("):src.index("umma_desc(")]


def test_no_cached_function_hands_out_device_tensors():
    """A tensor kept by a function for the whole process is made on one stream and read on others, and freed when the cache is full,
    with nothing to order it.  What is cached per function are plain host values."""
    import importlib
    import pkgutil

    import tace_b200

    cached = set()
    for info in pkgutil.walk_packages(tace_b200.__path__, "tace_b200."):
        if info.name.endswith(".libtace_b200"):  # the kernel library, not a Python module
            continue
        module = importlib.import_module(info.name)
        cached |= {f"{f.__module__}.{f.__name__}" for f in vars(module).values() if hasattr(f, "cache_info")}
    assert cached == {"tace_b200.graph._element_table", "tace_b200.graph._layout", "tace_b200.neighbour_list._workspace_bytes"}


def test_arrivals_of_the_tensor_core_gemms_order_memory():
    """What a role has read of a ring slot, a tile's description or an accumulator is overwritten by another role after the arrival that hands it
    back, so every such arrival has to order the reads before it; and nothing of the slot is read after it."""
    for name in ("tc_gemm.cu", "tc_gemm_fp16.cuh"):
        src = open(os.path.join(ROOT, "tace_b200", "csrc", name)).read()
        assert not re.search(r"mbarrier\.arrive[\w.]*\.relaxed", src), name
    epilogue = src[src.index("// -- epilogue"):src.index("tcgen05.dealloc")]
    after = epilogue[epilogue.index("mbar_arrive(info_empty(slot))"):]
    assert not re.search(r"\b(row_addr|row_top|info)\[", after)
