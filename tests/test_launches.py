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
