"""Barrier edges of the tensor-core kernels, read off their sources.

A wait that is missing between two roles of a CTA shows on the GPU only when the late role is
late, and running such a kernel there is a data race.  So the edges are checked in the text: in
the row-major kernels' MMA issuers every QK stands behind a wait for its K image, and every PV behind the
waits for its P and for its V image; in every loader a proxy fence stands between the wait for
a raw stage's readers, which read through the generic proxy, and the page copies, which write through
the async proxy.
"""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "pth_flash_attn_b200" / "csrc"
KERNELS = ["umma_rows_kernel.cu", "umma_rows2_kernel.cu", "umma_rows256_kernel.cu"]
WAIT = re.compile(r"wait_or_abort\w*\(&bars\[B::(\w+)")


def _code(name):
    text = (CSRC / name).read_text()
    text = re.sub(r"//[^\n]*", "", text)
    return text[text.index("__global__"):text.index("cudaError_t launch")]


def _role(code, warp):
    """The text of a role: from its branch to the next one."""
    start = re.search(rf"else if \(warp == k\w*{warp}\b", code).start()
    return code[start:code.index("else if (warp", start + 10)]


@pytest.mark.parametrize("name", KERNELS)
def test_every_mma_stands_behind_the_waits_for_its_operands(name):
    issuer = _role(_code(name), "MmaWarp")
    needs = {"issue_qk": {"kfull"}, "issue_pv": {"p_ready", "vfull"}}
    seen = set()
    waited = set()
    for token in re.finditer(WAIT.pattern + r"|\b(issue_qk|issue_pv)(?:_rows|_halves|_x|_w)\w*(?:<\w+>)?\(", issuer):
        barrier, issue = token.groups()
        if barrier:
            waited.add(barrier)
            continue
        seen.add(issue)
        assert needs[issue] <= waited, f"{name}: {issue} is issued without a wait for {sorted(needs[issue] - waited)}"
        waited -= needs[issue]
    assert seen == set(needs)


@pytest.mark.parametrize("name", KERNELS + ["umma_i8_kernel.cu"])
def test_page_copies_stand_behind_a_proxy_fence(name):
    loader = _role(_code(name), "LoadWarp")
    for copy in ("tma_load_3d(", "bulk_copy_g2s("):
        wait = re.search(r"(\w+)\(&bars\[B::raw_free", loader)
        assert wait and wait.start() < loader.index(copy)
        assert wait.group(1) == "wait_raw_free", f"{name}: {copy}) behind {wait.group(1)}"
    shared = (CSRC / "page_copy.cuh").read_text()
    body = shared[shared.index("bool wait_raw_free("):]
    body = body[:body.index("\n}")]
    assert body.index("wait_or_abort(") < body.index("fence_async_smem();") < body.index("return")


@pytest.mark.parametrize("name", KERNELS)
def test_the_scratch_copies_in_the_raw_ring_are_fenced(name):
    """query_start_loc and seq_lens are copied into the raw ring by plain stores before the first page copy."""
    code = _code(name)
    scratch = code[code.index("int* qsl_s = reinterpret_cast<int*>(smem + L::raw)"):code.index("resolve_row_tile(p, tile_index)")]
    last = scratch.rindex("__syncthreads();")
    assert scratch.index("resolve_row_tile_with(") < scratch.index("fence_async_smem();") < last


@pytest.mark.parametrize("name", KERNELS + ["umma_i8_kernel.cu"])
def test_no_mma_is_issued_behind_a_wait_that_gave_up(name):
    """Its operands are not what it needs, and nobody would wait for it before TMEM is freed."""
    code = _code(name)
    calls = [m.start() for m in re.finditer(r"\bif \([^;{}]*\belect_one\(\)\)\s*(?:\{|issue_pv\()", code)]
    assert len(calls) >= 2
    for at in calls:
        condition = code[at:code.index("elect_one()", at)]
        assert re.search(r"(\bok|\bgo|\bready|__all_sync\(0xffffffffu, sound\)) &&", condition), f"{name}: {condition}"
    if "sound" in code:
        assert "const bool sound = ok && *abort_flag == 0;" in code


@pytest.mark.parametrize("name", KERNELS)
def test_tmem_is_freed_before_the_wait_for_the_integer_kernel(name):
    """That kernel lets this one start before it allocates: a CTA that waited for it and held TMEM would hold it up for good."""
    code = _code(name)
    code = code[code.index("if (!p.late_wait) pdl_wait();"):]
    waits = [m.start() for m in re.finditer(r"if \(p\.late_wait\) pdl_wait\(\);", code)]
    frees = [m.start() for m in re.finditer(r"tmem_dealloc\(", code)]
    assert len(waits) == len(frees) == 2        # without work, and at the end
    assert frees[0] < waits[0] < frees[1] < waits[1]


@pytest.mark.parametrize("name", KERNELS)
def test_a_cta_of_an_unused_piece_leaves_without_tmem(name):
    """Most pieces of a generous bound are not used, and taking TMEM for them cost small launches 5 %."""
    code = _code(name)
    assert code.count("const bool tmem_ahead = split == 0;") == 1
    allocs = [m.start() for m in re.finditer(r"tmem_alloc\(tslot, 512\)", code)]
    frees = [m.start() for m in re.finditer(r"tmem_dealloc\(", code)]
    found = code.index("item = *reinterpret_cast<const RowsItem*>(item_s);")
    later = code.index("if (!tmem_ahead) {")
    assert len(allocs) == len(frees) == 2
    assert "if (tmem_ahead) {" in code[:allocs[0]] and allocs[0] < found < frees[0] < later < allocs[1] < frees[1]
    assert re.search(r"if \(tmem_ahead && warp == k\wLoadWarp\) tc::tmem_dealloc\(", code[found:later])
    # its address is read by everybody: a barrier of the CTA behind the allocation, between the two TMEM fences
    behind = code[allocs[1]:code.rindex("tmem_base = *tslot;")]
    assert behind.index("fence_before_sync();") < behind.index("__syncthreads();") < behind.index("fence_after_sync();")
