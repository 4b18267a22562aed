"""Who may let the next kernel start early (programmatic dependent launch), checked on the sources: the races this rules out
need particular timing to show on a device.

A kernel may read before its own wait what the kernel in front of it does not write (a product's weights, a routing plan,
operands the caller declared static). What it reads must then be complete when the kernel in front lets it start: so the
expert path's kernels wait before their trigger, and a quantiser has no trigger unless the product directly behind it
holds back its own dependents until the quantiser has finished."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "gpu_kernels_b200" / "csrc"
WAIT = r"(?:ptx::)?grid_dependency_wait\(\);"
TRIGGER = r"(?:ptx::)?grid_launch_dependents\(\);"


def code(name):
    lines = (re.sub(r"//.*", "", line).strip() for line in (CSRC / name).read_text().splitlines())
    return "\n".join(line for line in lines if line)


def first_statements(text, kernel):
    body = re.search(r"\b" + kernel + r"\s*\([^{;]*\)\s*\{\n((?:.*\n){2})", text)
    assert body, kernel
    return body.group(1)


def chained_kernels(text):
    """Kernels that reach launch_chained() by name or through a local lambda that is given the kernel."""
    return (set(re.findall(r"launch_chained\((\w+?)(?:<[^>]*>)?,", text)) - {"kernel"}) | set(re.findall(r"\bgo\((\w+)<", text))


def test_chain_point_waits_first():
    assert re.search(r"void chain_point\(\) \{\n" + WAIT + "\n" + TRIGGER + r"\n\}", code("ptx.cuh"))
    for path in CSRC.iterdir():
        if path.suffix in (".cu", ".cuh", ".h") and path.name != "ptx.cuh":
            assert "griddepcontrol" not in code(path.name), f"{path.name}: raw instruction"


def test_expert_path_kernels_wait_first():
    text = code("nvfp4_moe.cu")
    kernels = chained_kernels(text)
    assert {"plan_kernel", "pack_kernel", "swiglu_quant_kernel", "quantise_route_kernel", "reduce_kernel"} <= kernels
    for kernel in kernels:
        assert first_statements(text, kernel).startswith("ptx::chain_point();"), kernel
    assert not re.search(TRIGGER, text)


@pytest.mark.parametrize("kernel,trigger", [("quantise_kernel", "if constexpr (EARLY) ptx::grid_launch_dependents();"), ("quantise_mx_kernel", None)])
def test_quantisers_let_nothing_start_early_by_themselves(kernel, trigger):
    text = code("nvfp4_quant.cu")
    assert kernel in chained_kernels(text)
    first, second = first_statements(text, kernel).splitlines()
    assert re.fullmatch(WAIT, first)
    assert second == trigger if trigger else "dependents" not in second
    assert re.findall(r".*" + TRIGGER, text) == ["if constexpr (EARLY) ptx::grid_launch_dependents();"]
    # early: only for the linear call, whose product is launched with late_trigger
    assert re.findall(r"(.*)launch_quantise<\w+, true>\(", text) == ["if (early) "]
    capi = code("nvfp4_capi.cu")
    calls = re.findall(r"nvfp4_b200::quantise\(x(?:[^;]*\n?)*?;", capi)
    early = [c for c in calls if re.search(r"true\s*\)\s*;$", c)]
    assert len(calls) == 2 and len(early) == 1
    behind = capi[capi.index(early[0]):]
    assert behind.index("q.late_trigger = 2;") < behind.index("p.impl.launch(q,")


def test_a_product_that_triggers_late_waits_first():
    text = code("nvfp4_gemm.cu")
    triggers = re.findall(r".*\n.*" + TRIGGER, text)
    assert len(triggers) == 4
    assert sum("if (threadIdx.x == 0 && !g.late_trigger)" in t for t in triggers) == 1
    after_wait = [t for t in triggers if re.search(r"if \(g\.late_trigger(?: == 1)? && threadIdx\.x == 0\)", t)]
    assert len(after_wait) == 2 and all(re.match(r".*" + WAIT, t) for t in after_wait)
    # the producer's: behind its last load, and release_held waits before its first load of A
    last = [t for t in triggers if "g.late_trigger == 2" in t]
    assert len(last) == 1 and last[0].startswith("if (early_b && issued < Cfg::STAGES) release_held(") and "\nif (early_b && " in last[0]
    assert re.search(r"void release_held\([^{]*\{\n" + WAIT, text)
    assert "g.late_trigger = p.late_trigger;" in text and "g.static_operands = g.late_trigger =" in text
