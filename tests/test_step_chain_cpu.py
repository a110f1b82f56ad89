"""Kernels of a programmatically launched chain may be resident while earlier
launches still write.  Read-only loads (__restrict__ inputs, __ldg, __ldcg) are
for what was complete before the chain began; the first launch is an ordinary one."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "btorch_b200" / "csrc"
# indices, weights and inputs that no launch of a chain writes
CONSTANT = {"ptr", "col", "wts", "csr_ptr", "csr_dst", "csc_ptr", "csc_src", "w", "x", "perm", "z_given"}
KERNEL = re.compile(r"__global__\s+void\s+(?:__launch_bounds__\([^{;]*?\)\s*)?(k_\w+)\(([^{;]*)\)\s*\{(.*?)\n\}", re.S)


def chain_kernels():
    out = []
    for path in sorted(CSRC.glob("*.cu")):
        for m in KERNEL.finditer(path.read_text()):
            if re.search(r"step_(begin|wait)\(\);", m.group(3)):
                out.append(pytest.param(m.group(2), m.group(3), id=m.group(1)))
    return out


def test_every_chain_kernel_is_seen():
    text = "".join(p.read_text() for p in CSRC.glob("*.cu"))
    assert len(chain_kernels()) == len(re.findall(r"step_(?:begin|wait)\(\);", text)) >= 9


@pytest.mark.parametrize("params,body", chain_kernels())
def test_read_only_inputs_are_constant_over_the_chain(params, body):
    names = set(re.findall(r"__restrict__\s+(\w+)", params))
    assert names <= CONSTANT
    assert "__ldcg(" not in body
    assert set(re.findall(r"__ldg\((?:reinterpret_cast<[^>]*>\()?(\w+)", body)) - {"__ldg"} <= CONSTANT
    assert "__restrict__" not in body


def test_chains_start_with_an_ordinary_launch():
    firsts = {p.name: re.findall(r"launch_step\((k == 0|first|false|true), ", p.read_text()) for p in CSRC.glob("*.cu")}
    calls = {p.name: p.read_text().count("launch_step(") for p in CSRC.glob("*.cu")}
    for name, n in calls.items():
        named_in_comments = len(re.findall(r"//.*launch_step\(", (CSRC / name).read_text()))
        assert len(firsts[name]) == n - named_in_comments, name
    assert firsts["engine.cu"].count("k == 0") == 3


def test_transposed_operand_is_read_by_plain_loads():
    text = (CSRC / "spmm.cu").read_text()
    body = text[text.index("FVec<V> ld_vec("):]
    assert "__ldg" not in body[: body.index("\n}")]
    rows = text[text.index("void rows_gather("):]
    assert set(re.findall(r"__restrict__\s+(\w+)", rows[: rows.index("{")])) <= CONSTANT
