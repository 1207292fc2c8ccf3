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


ROLE = re.compile(r"// -{8,} *(?P<name>[^-\n]+?) *-{8,}")
RELEASE = re.compile(r"umma_commit\(&(?P<ring>\w+)_empty\[")
# ring slots that a thread releases without having waited for them, and why they are full
IMPLIED = {("flash_attn_bwd.cu", "accumulating products", "y1"):
           "dS follows S, which was formed from the slot"}


def unwaited(name, source):
    """(role, ring) where the thread whose products release a ring's slots never waits for them to be full.
    Roles are the stretches between dashed comments; a ring chosen at run time (``y_full``) goes by its
    first letter."""
    source = source.replace("\\\n", " ")
    heads = list(ROLE.finditer(source))
    found = []
    for head, after in zip(heads, heads[1:] + [None]):
        body = source[head.end():after.start() if after else len(source)]
        for ring in sorted(set(m["ring"] for m in RELEASE.finditer(body))):
            waits = (f"mbar_wait(&{ring}_full[", f"mbar_wait(&{ring[0]}_full[", f"mbar_wait({ring}_full")
            if not any(w in body for w in waits) and (name, head["name"], ring) not in IMPLIED:
                found.append((head["name"], ring))
    return found


def test_the_reader_of_roles_sees_what_it_should():
    role = "// ---------- one ----------\n%s\n// ---------- two ----------\nmbar_wait(&y2_full[0]);"
    assert unwaited("x", role % "umma_commit(&y2_empty[s]);") == [("one", "y2")]
    assert unwaited("x", role % "mbar_wait(&y2_full[s]); umma_commit(&y2_empty[s]);") == []
    assert unwaited("x", role % "mbar_wait(&y_full[s]); umma_commit(&y2_empty[s]);") == []


@pytest.mark.parametrize("name", ["flash_attn.cu", "flash_attn_bwd.cu"])
def test_a_thread_waits_for_what_its_products_read(name):
    with open(os.path.join(CSRC, name)) as f:
        source = f.read()
    assert len(RELEASE.findall(source)) >= 3
    missing = unwaited(name, source)
    assert not missing, f"{name}: slots released without a wait for their loads: {missing}"


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
