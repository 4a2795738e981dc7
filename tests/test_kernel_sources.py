"""What a kernel's source has to hold that no run shows: read as text, nothing is compiled."""
import glob
import os
import re

from idempotent_llm_b200.kernels import ops

CSRC = os.path.join(os.path.dirname(ops.__file__), "..", "csrc")


def _kernels():
    """(file, name, body) of every kernel."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__ void\s+(?:__launch_bounds__\([^{;]*?\)\s+)?(\w+)\s*\(", text):
            at = text.index("{", m.end())
            depth, end = 1, at + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield os.path.basename(path), m.group(1), text[at:end]


def test_the_next_kernel_starts_only_behind_an_allocation_of_tensor_memory():
    """A block of the next kernel that starts beside one that has not got its columns yet can take them, and keeps them until the kernel
    before has ended: neither goes on.  So a kernel that allocates lets the next one start behind the barrier behind the allocation."""
    seen = []
    for file, name, body in _kernels():
        alloc = re.search(r"\btmem_alloc(_pair)?\(", body)
        if not alloc:
            continue
        seen.append(name)
        starts = [m.start() for m in re.finditer(r"\bpdl_launch_dependents\(", body)]
        if not starts:
            continue                                     # (lets nothing start before its end)
        barrier = body.find("__syncthreads()", alloc.end())
        assert barrier > 0 and min(starts) > barrier, f"{file}: {name}"
    assert {"attention_tc_kernel", "gemm_persistent_kernel", "gemm_experts_kernel", "gemm_pair_kernel", "gemm_qkv_tokens_kernel",
            "gemm_small_kernel", "gemm_wide_kernel", "gemm_f32_split_kernel", "gemm_f32_wide_kernel"} <= set(seen), seen


def test_uploads_are_refused_under_capture(monkeypatch):
    """A captured copy would be made again from host memory that is gone by then (the copy does not wait, so nothing else refuses it)."""
    import pytest
    import torch
    K = ops.Kernels.__new__(ops.Kernels)
    K.device = torch.device("cpu")
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    assert K._uploaded([3, 1, 2]).tolist() == [3, 1, 2]
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    with pytest.raises(ops.KernelError, match="capture"):
        K._uploaded([3, 1, 2])
