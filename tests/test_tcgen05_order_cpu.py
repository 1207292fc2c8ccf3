"""Order of tensor-memory accesses against barriers, read off the kernel sources.

An mbarrier wait alone does not order ``tcgen05`` instructions behind it: a thread that accesses
tensor memory (``tcgen05.ld`` / ``st`` / ``mma``) after waiting for another thread or for a commit
executes ``tcgen05.fence::after_thread_sync`` (``fence_after_sync``) in between."""
import os
import re

import pytest

import slapo_b200

CSRC = os.path.join(os.path.dirname(slapo_b200.__file__), "csrc")
KERNELS = ["flash_attn.cu", "flash_attn_bwd.cu", "gemm.cu", "gemm2.cu", "comm_gemm.cu"]
EVENT = re.compile(r"(?P<wait>\bmbar_wait(?:_warp)?\()|(?P<fence>\bfence_after_sync\(\))"
                   r"|(?P<access>\b(?:tmem_ld_x|tmem_st_x|umma_f16|scores\(|accumulate\()\w*)"
                   r"|(?P<open>\{)|(?P<close>\}(?P<more>\s*else\b)?)")


def unfenced(source):
    """Line numbers of accesses with a wait, and no fence on every path, before them.  A block
    that may be skipped fences nothing behind it; an ``else`` starts from where its ``if`` did."""
    source = re.sub(r"//[^\n]*", "", source)
    found, waited, blocks, carry = [], False, [], None
    for m in EVENT.finditer(source):
        if m["wait"]:
            waited = True
        elif m["fence"]:
            waited = False
        elif m["access"]:
            if waited:
                found.append(source.count("\n", 0, m.start()) + 1)
        elif m["open"]:
            # (state at its start, state of the paths around it)
            blocks.append((waited, waited if carry is None else carry))
            carry = None
        else:
            start, around = blocks.pop()
            if m["more"]:
                carry, waited = waited or around, start
            else:
                waited = waited or around
    return found


def test_the_reader_sees_what_it_should():
    assert unfenced("{ mbar_wait(a); tmem_ld_x32(r); }") == [1]
    assert unfenced("{ mbar_wait(a); fence_after_sync(); tmem_ld_x32(r); }") == []
    assert unfenced("{ mbar_wait(a);\nif (x) { fence_after_sync(); }\ntmem_st_x16(r); }") == [3]
    assert unfenced("{ if (x) { mbar_wait(a); } else { umma_f16(d); } }") == []
    assert unfenced("{ if (x) { mbar_wait(a); } else { y; }\numma_f16(d); }") == [2]
    assert unfenced("{ if (!mbar_wait(a)) { break; } fence_after_sync(); scores(x); }") == []


@pytest.mark.parametrize("name", KERNELS)
def test_tensor_memory_accesses_follow_the_fence(name):
    with open(os.path.join(CSRC, name)) as f:
        lines = unfenced(f.read())
    assert not lines, f"{name}: tensor memory accessed after a wait without the fence at {lines}"
