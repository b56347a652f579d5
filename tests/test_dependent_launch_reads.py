"""Kernels launched on the tail of the kernel before them (programmatic dependent
launch) read what that kernel writes with plain loads only: a const __restrict__
parameter and __ldg promise the compiler that the memory does not change while the
kernel runs, so such a load may be moved over the wait."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "dynamicradiancevolume_gb300" / "csrc"
WAIT = re.compile(r"griddepcontrol\.wait|pdl_wait_and_release\(\);")
KERNEL = re.compile(r"__global__\s+void\s+(?:__\w+\([^()]*\)\s*)*(\w+)\s*\(([^{;]*?)\)\s*\{")


def _kernels():
    for f in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        starts = list(KERNEL.finditer(text))
        for m, n in zip(starts, starts[1:] + [None]):
            yield f.name, m.group(1), m.group(2), text[m.end():n.start() if n else len(text)]


def test_waiting_kernels_take_no_read_only_parameters():
    waiting = [(f, k, params) for f, k, params, body in _kernels() if WAIT.search(body)]
    assert {"adam_kernel", "gather_kernel", "cone_kernel", "apply_kernel"} <= {k for _, k, _ in waiting}
    bad = [(f, k) for f, k, params in waiting if re.search(r"const\s+\w+\s*\*\s*__restrict__", params)]
    assert not bad, bad


def test_pair_list_fields_of_the_kernel_before_are_read_plainly():
    """The pair list's cache and block arrays are the cull's, complete before any
    later pass starts; the other fields are written by the pass before their reader."""
    bad = [(f, k) for f, k, _, body in _kernels()
           if re.search(r"__ldg\(\s*L\.(shadow|partials|units|unit_range|order|cls|counters|info)\b", body)]
    assert not bad, bad
