"""What a kernel may do before the one ahead of it on the stream has finished, read from the sources: the failures these
rules prevent (a race on memory, two kernels that wait for each other) are not for running."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "mamba_trainer_b200" / "csrc"


def _text(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def _kernels():
    """name -> body of every __global__ function."""
    found = {}
    for path in sorted(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh"))):
        s = _text(path)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", s):
            at = s.index("{", m.end())
            depth, end = 0, at
            while True:
                depth += {"{": 1, "}": -1}.get(s[end], 0)
                end += 1
                if depth == 0:
                    break
            found[m.group(1)] = s[at:end]
    return found


def test_kernels_launched_early_wait_before_they_touch_memory():
    kernels = _kernels()
    launched = set()
    for path in CSRC.glob("*.cu"):
        s = _text(path)
        # kernels named in the statement of a launch, or chosen for its `kern` above it
        for text in re.findall(r"\blaunch\(([^;]*);", s) + re.findall(r"auto kern\s*=([^;]*);", s):
            launched |= set(re.findall(r"\w+", text)) & set(kernels)
    assert {"tc_fwd_kernel", "tc_bwd_kernel", "k_step_rows", "k_group_state", "k_rows_adjoint", "k_front_bwd", "k_gate_bwd",
            "kb_final"} <= launched
    for name in launched:
        before, wait, _ = kernels[name].partition("after_predecessor()")
        assert wait, name
        # set-up of shared memory may come first; global memory, bulk copies and TMEM may not
        assert not re.search(r"tmem_alloc|bulk_|tma_|__ldg|__ldcg|atomic|prefetch|ld_volatile", before), name
