"""The GKR prover's launches are programmatic dependents: a kernel runs beside the one before it until it
waits for that one's end. Before the wait it may touch its own shared memory and what no launch of the
chain writes (the table of layer columns and the counts), nothing else. Checked on the kernels' source."""
import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parent.parent / "proving_gb300" / "csrc" / "gkr_prove.cu").read_text()
CONSTANT = {"cols", "n_inst", "n_layers"}
KERNELS = re.findall(r"__global__ void __launch_bounds__\(\w+\)\s+(gkr_\w+)\((.*?)\n}\n", SOURCE, re.S)


def test_the_chain_is_found():
    assert {name for name, _ in KERNELS} == {"gkr_round_kernel", "gkr_tail_kernel", "gkr_start_kernel"}


@pytest.mark.parametrize("name,body", KERNELS, ids=[name for name, _ in KERNELS])
def test_nothing_written_by_the_chain_is_touched_before_the_wait(name, body):
    before, wait, _ = body.partition("chain_wait();")
    assert wait, f"{name} never waits"
    assert set(re.findall(r"\bg\.(\w+)", before)) <= CONSTANT


def test_the_constant_tables_are_never_written():
    assert re.search(r"const LayerCols\* cols;", SOURCE)
    assert not re.search(r"const_cast<LayerCols|copy_words\([^;]*g\.cols", SOURCE)
