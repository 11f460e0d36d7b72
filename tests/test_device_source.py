"""Orderings in the device and host sources that no run can be relied on to
show: a missing memory barrier between lanes, a call on the wrong device, an
optional allocation ahead of one that has to succeed."""
from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "zillumgl_gb300" / "csrc"


def _body(name: str, head: str) -> str:
    """The braces behind the first occurrence of `head`, comments left out."""
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    start = text.index("{", text.index(head))
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError(f"{name}: unbalanced braces behind {head}")


def test_subtree_bins_are_read_behind_a_barrier():
    """The lanes of a warp fill the bins with shared-memory atomics; a warp
    reduction does not order them before other lanes' plain reads."""
    body = _body("bvh_build_gpu.cu", "subtree_kernel(")
    filled = max(m.end() for m in re.finditer(r"atomic\w+\(&ws\.", body))
    read = re.search(r"=\s*ws\.(lo|hi|cnt)\[bb\]", body).start()
    assert filled < read
    assert "__syncwarp();" in body[filled:read]


def test_staged_calls_take_their_turn():
    """Two calls of one handle at once would append to the same lists, beyond
    their ends; the batched renderer's run on its own stream."""
    for name, heads in (("render.cu", ("void staged_passes(", "void staged_light(")),
                        ("render_diff.cu", ("zgl_status zgl_diff_forward(", "zgl_status zgl_diff_backward("))):
        for head in heads:
            body = _body(name, head)
            launch = re.search(r"ZGL_CUDA\(launch_(staged|staged_light|replay)\(", body).start()
            assert re.search(r"const StagedTurn turn\((it|d)->pool, st\);\s*$", body[:launch]), head
        text = (CSRC / name).read_text()
        assert len(re.findall(r"ZGL_CUDA\(launch_(?:staged|staged_light|replay)\(", text)) == len(heads)


def test_export_runs_on_the_accelerators_device():
    """An export allocates and launches; the current device may be another one
    than the tree's, as in the trace calls."""
    for entry in ("zgl_accel_export", "zgl_trace_closest", "zgl_trace_any", "zgl_trace_count",
                  "zgl_trace_closest_noalloc"):
        body = _body("accel.cu", f"zgl_status {entry}(")
        guard = body.find("DeviceGuard dg(accel->device);")
        work = re.search(r"export_device_tree\(|launch_trace_|Staging st\(|cudaMemcpy", body).start()
        assert 0 <= guard < work, entry


def test_optional_memory_comes_last():
    """The staged renderers run without their pool: it is taken behind all that
    a handle cannot do without, and given back where that is short."""
    for name, entry in (("render_diff.cu", "zgl_diff_create"), ("render_batch.cu", "zgl_batch_create")):
        body = _body(name, f"zgl_status {entry}(")
        needed = max(m.start() for m in re.finditer(r"ZGL_CUDA\(cudaMalloc\(|ZGL_CUDA\(cudaEventCreate", body))
        assert needed < body.index("staged_alloc("), entry
    for name, entry, array in (("render_diff.cu", "zgl_diff_step_l2", "d_dimage"),
                               ("render.cu", "zgl_integrator_render_passes", "d_passes")):
        body = _body(name, f"zgl_status {entry}(")
        assert re.search(rf"staged_malloc_beside\(\w+->pool, \(void\*\*\)&\w+->{array}", body), entry


def test_export_needs_no_device_memory():
    """An export without memory to spare rearranges the records on the host."""
    body = _body("wide_build.cu", "void export_device_tree(")
    assert "ZGL_ERR_OOM" not in body and "return export_on_host(" in body[body.index("cudaMalloc("):]
