"""What no run can show to be missing, looked for in the source: orders of memory,
and lanes of a warp that have to agree.

sstep_kernel and ku_rest_kernel write global arrays and march them in the same
launch, and march several units whose shared memory is laid out differently.
Bulk copies (the async proxy) are ordered after ordinary accesses only by a
proxy fence on the way from the one to the other."""
import os
import random
import re
from fractions import Fraction

import komegafoulingmodel_b200

CSRC = os.path.join(os.path.dirname(komegafoulingmodel_b200.__file__), "csrc")
FENCE = "ss_proxy_fence();"


def body(name, file="kofm_sstep.cuh"):
    """The body of a device function, without comments."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, file)).read())
    at = re.search(r"__device__[^;{}]*\b%s\([^;{}]*\)\s*\{" % name, text)
    depth, i = 1, at.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
    return text[at.end():i - 1]


def test_the_fences_cover_global_and_shared_memory():
    assert 'asm volatile("fence.proxy.async;" ::: "memory")' in body("ss_proxy_fence")
    assert 'asm volatile("fence.proxy.async.shared::cta;" ::: "memory")' in body("ss_proxy_fence_shared")


def test_grid_barrier_orders_writes_before_later_copies():
    sync = body("ss_sync")
    assert FENCE in sync[:sync.index("atomicAdd")], "before the arrival"
    assert FENCE in sync[sync.rindex("ss_sync_march();"):], "after the wait"


def test_a_unit_ends_with_a_fence():
    march = body("ss_march")
    assert re.search(r"ss_proxy_fence_shared\(\);\s*ss_sync_march\(\);\s*$", march)
    assert "ss_proxy_fence_shared();" in body("ss_unit_sums")[-40:]


def test_only_constant_arrays_are_read_non_coherently():
    """k, omega and the rows change within ku_rest_kernel; the flags and the index
    of the link fractions do not."""
    for name, file in (("km_assemble", "kofm_komega.cuh"), ("ss_resid_units", "kofm_sstep.cuh"),
                       ("ss_write_units", "kofm_sstep.cuh"), ("ss_march", "kofm_sstep.cuh")):
        for args in re.findall(r"__ldg\(([^)]*)", body(name, file)):
            assert args.startswith(("p.ntype", "p.dxidx")), (name, args)


def test_overlapped_kernels_read_behind_their_wait():
    """A kernel placed while its predecessor runs: what that one wrote is read
    through ordinary loads, which stay below the wait, or through a pointer taken
    behind it."""
    step = body("lb_block", "kofm_lb.cuh")
    assert "if constexpr (!KOMEGA && !NEQ) grid_wait();" in open(os.path.join(CSRC, "kofm_lb.cuh")).read()
    assert re.findall(r"load4<([^>]*)>", step) == ["KOMEGA || NEQ"] * 2
    # the other read-only loads of the collide: the FP16_NEQ moments, wall distances
    assert re.findall(r"(\w*ldg\w*)\(", step) == ["fld_ldg4"]
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "kofm_adjoint.inc")).read())
    for name, pointers in (("k_adj_lambda", ("nu", "lam", "sg")), ("k_adj_stream_t", ("lam", "nu", "dq"))):
        kernel = text[text.index(name + "("):]
        kernel = kernel[kernel.index("{"):]
        waits = re.match(r"\{\s*grid_wait\(\);((?:\s*after_wait\(\w+\);)*)", kernel).group(1)
        assert re.findall(r"\((\w+)\)", waits) == list(pointers), name


def test_lanes_agree_on_what_their_branches_read():
    """The tests that end a cycle are taken by every lane of a warp from its own
    copy of a sum over the lanes; with that sum's first addition fused into the
    product before it, lanes i and j round a_i b_i + a_j b_j differently, and the
    warp could part at a shuffle that waits for all of it."""
    def fma(a, b, c):
        return float(Fraction(a) * Fraction(b) + Fraction(c))

    rng = random.Random(1)
    draw = [[rng.uniform(0.5, 1.0) for _ in range(4)] for _ in range(100)]
    assert any(fma(a, b, c * d) != fma(c, d, a * b) for a, b, c, d in draw)
    assert all(a * b + c * d == c * d + a * b for a, b, c, d in draw)
    assert "x = __dadd_rn(x, __shfl_xor_sync(0xffffffffu, x, off));" in body("ss_sum16")


def test_a_block_outlives_the_copies_of_a_failed_wait():
    """A wait that ran out may leave bulk copies in flight into the block's shared
    memory; the block ends only some time after its last one."""
    end = body("ss_specialise")
    end = end[end.rindex("ss_sync_block();"):]
    assert re.search(r"if \(\*\(volatile int\*\)&ss_sm\(\)\.dead\)\s*for \(int i = 0; i < 1000; \+\+i\) __nanosleep\(1000\);", end)
