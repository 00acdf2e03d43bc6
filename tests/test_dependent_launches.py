"""Kernels that start while the stream's last kernel still runs: the rules stated
at launch_dependent, checked in the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "hawkes_b200", "csrc")
WAIT, TRIGGER = "cudaGridDependencySynchronize()", "cudaTriggerProgrammaticLaunchCompletion()"


def _kernels():
    """(name, parameters, body) of every kernel in the sources, comments removed."""
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh", ".inc")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?"
                             r"(\w+)\s*\(([^)]*)\)\s*\{", text):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield m.group(1), m.group(2), text[m.end():end]


def test_dependent_kernels_make_no_promise_about_memory_still_written():
    waiting = {name: par for name, par, body in _kernels() if WAIT in body}
    assert {"sweep_f64_list_kernel", "sweep_f32c_list_kernel", "finish_list_kernel",
            "mh_step_kernel"} <= set(waiting)
    for name, par in waiting.items():
        assert "__restrict__" not in par, name


def test_the_next_kernel_is_allowed_after_the_wait_only():
    sources = "".join(open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC))
                      if f.endswith((".cu", ".cuh", ".inc")))
    triggering = [(name, body) for name, _, body in _kernels() if TRIGGER in body]
    assert len(triggering) >= 5
    for name, body in triggering:
        if WAIT in body:
            assert body.index(WAIT) < body.index(TRIGGER), name
        else:  # launched in stream order
            assert re.search(rf"\b{name}(<[^<>;]*>)?<<<", sources), name
            for call in re.findall(r"launch_dependent\((?:[^()]|\([^()]*\))*\)", sources):
                assert name not in call, name


def test_data_other_blocks_wrote_is_read_past_the_read_only_path():
    text = open(os.path.join(CSRC, "hphc_kernels.cu")).read()
    total = text[text.index("bool finish_total("):]
    total = total[:total.index("\n}\n")]
    assert "const volatile double* sums" in total and "__restrict__" not in total
