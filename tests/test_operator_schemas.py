"""What the operators declare to write, on the CPU: a tracer that trusts a schema takes an operator without such a mark for pure."""
import pytest
import torch

from warpstate_ai_b200.ops import _ext


@pytest.fixture(scope="module")
def schemas():
    if not _ext.load():
        pytest.skip("the kernel library cannot be built here")
    return [s for s in torch._C._jit_get_all_schemas() if s.name.startswith("ws_b200::")]


def written(argument):
    return argument.alias_info is not None and argument.alias_info.is_write


def test_error_words_are_written(schemas):
    found = [(s.name, a) for s in schemas for a in s.arguments if a.name in ("error_flag", "status") and "Tensor" in str(a.type)]
    assert len(found) > 10
    reads = {"ws_b200::grad_norm_clip", "ws_b200::clip_from_partials"}      # their status is an input
    assert [name for name, a in found if not written(a) and name not in reads] == []


def test_a_native_block_writes_its_weights_gradients(schemas):
    block, = (s for s in schemas if s.name == "ws_b200::block")
    assert [a.name for a in block.arguments if written(a)] == ["main", "error_flag"]
