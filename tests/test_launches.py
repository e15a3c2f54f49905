"""How the library's sources launch kernels (read as text: no device).

A launch may be refused (its configuration, its resources).  Then the kernels behind
it work on what an earlier call left, so every launch's status has to reach the caller."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "unicycle_b200", "csrc")


def _sources():
    for p in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = open(p).read()
        yield os.path.basename(p), re.sub(r"//[^\n]*|/\*.*?\*/", lambda m: re.sub(r"[^\n]", " ", m.group()), text,
                                          flags=re.S)


def test_every_launch_status_is_used():
    """A programmatic launch, and each function that hands one on, as a statement of
    its own would drop its status."""
    names = r"launch_pdl|launch_traction(?:_t)?|launch_products|hmatrix_products|hmatrix_apply|enqueue_stage|" \
            r"enqueue_attempt(?:_raw)?|rk_enqueue_\w+|launch_hpass|launch_hier|launch_contract|launch_all"
    found = 0
    for name, text in _sources():
        found += len(re.findall(rf"\b(?:{names})\b\s*(?:<[^;()]*>)?\(", text))
        for m in re.finditer(rf"(?:^|[;{{}}\)]|\belse)\s*(?:{names})\b\s*(?:<[^;()]*>)?\(", text, flags=re.M):
            line = text[:m.end()].count("\n") + 1
            raise AssertionError(f"{name}:{line}: the launch's status is dropped")
    assert found > 20


def test_no_read_only_loads_in_the_stage_kernels():
    """The launches of rk.cu overlap: one starts while the one in front still writes
    the rates and partial sums that it reads after its wait.  A load on the read-only
    path may return an older value."""
    text = dict(_sources())["rk.cu"]
    assert "launch_pdl(" in text
    assert not re.findall(r"__ldg\s*\(|ld\.global\.nc", text)


def test_overlapping_kernels_promise_read_only_memory_for_tables_alone():
    """Kernels launched programmatically start while the one in front runs.  What they
    read through `const ... __restrict__` (which lets the compiler take the read-only
    path) or __ldg has to be laid out once: K, its scales, plans and index tables."""
    tables = {"K", "scale", "tiles", "segs", "cta_seg", "units", "zu", "pws", "A"}
    kernels, text = set(), ""
    for _, t in _sources():
        kernels |= {k for m in re.finditer(r"\blaunch_pdl\(([^;]*)", t) for k in re.findall(r"\bk_\w+", m.group(1))}
        text += t
    kernels |= {"k_traction"}    # launched through a variable
    assert len(kernels) == 12
    for k in kernels:
        m = re.search(rf"__global__[^;{{}}]*?\b{k}\s*\(([^{{}}]*?)\)\s*{{", text)
        assert m, k
        named = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", m.group(1)))
        assert named <= tables, (k, named - tables)
    ens = dict(_sources())["ensemble.cu"]
    assert set(re.findall(r"__ldg\(\s*(\w+)", ens)) <= {"ubidx"}


def test_traction_kernel_reads_the_control_block_once():
    """The warps of a CTA wait for one another at named barriers, without a limit: they
    have to agree on whether there is anything to do, so one thread reads the control
    block for all of them (another CTA may change it between two reads)."""
    text = dict(_sources())["rk.cu"]
    m = re.search(r"__global__[^;{}]*?\bk_traction\b.*?\n}\n", text, flags=re.S)
    body = m.group()
    assert not re.findall(r"\bctl_live\(|ctl->(?:active|need_stage1|wait_ns|h)\b", body)
    assert body.count("tm_head(") == 2 and "&head_read" in body
