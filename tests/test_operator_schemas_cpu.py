"""What the operators declare: an argument that a call writes has to say so, or a tracer may reorder or drop the call."""
import pytest
import torch

from gpu_ipc_example_b200._ext import load


@pytest.mark.parametrize("name,written", [
    ("rope_decode_attention", {"kcache", "vcache", "workspace"}),
    ("decode_step", {"h", "kcache", "vcache", "workspace"}),
])
def test_written_arguments_are_declared(name, written):
    load()
    schema = getattr(torch.ops.b200ipc, name).default._schema
    assert {a.name for a in schema.arguments if a.alias_info is not None and a.alias_info.is_write} == written
