"""What the Python layer refuses before a kernel is launched.  The library is a stand-in that counts calls: nothing here needs a GPU."""
import dataclasses
import subprocess
import sys

import pytest
import torch

from tlaloc_b200 import ops
from tlaloc_b200.attrs import PagedAttentionShape, parse_paged_attention


@pytest.fixture
def calls(monkeypatch):
    """The C functions that were called."""
    seen = []

    class Library:
        def __getattr__(self, name):
            return lambda *args: seen.append(name) or 0

    monkeypatch.setattr(ops.N, "lib", lambda: Library())
    return seen


def test_rows_on_the_host_are_refused(calls, monkeypatch):
    """latent_kv_write has no other look at where its rows lie than the stream of their device."""
    monkeypatch.setattr(ops, "_dev", lambda *ts: None)  # the other operands are on the device
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 0, raising=False)
    i32 = dict(dtype=torch.int32)
    low, pool, table = torch.zeros(2, 12), torch.zeros(1, 16, 12), torch.zeros(3, 2)
    with pytest.raises(ValueError, match="CUDA"):
        ops.latent_kv_write(low, None, torch.ones(8), 1e-5, torch.zeros(2, **i32), table, table, torch.zeros(2, **i32), None, pool, q_rank=0, kv_rank=8, rot_dim=4, rot_dims=4)
    assert calls == []


def test_a_torch_without_cuda_imports_the_operators():
    program = "import torch; del torch._C._cuda_getCurrentRawStream; import tlaloc_b200.ops, tlaloc_b200.decoder, tlaloc_b200.latent_decoder, tlaloc_b200.mixed_decoder"
    done = subprocess.run([sys.executable, "-c", program], capture_output=True, text=True)
    assert done.returncode == 0, done.stderr


def on_the_device(*shape):
    """A tensor that says it is on a CUDA device."""
    class Tensor(torch.Tensor):
        is_cuda = True

    return torch.zeros(shape).as_subclass(Tensor)


@pytest.mark.parametrize("name", ["x", "out", "residual"])
@pytest.mark.parametrize("shape", [(), (4,), (1, 2, 4)])
def test_a_projection_names_the_operand_of_another_rank(calls, name, shape):
    operands = {n: on_the_device(2, 4) for n in ("x", "out", "residual")}
    operands[name] = on_the_device(*shape)
    with pytest.raises(ValueError, match=f"DENSE_PROJ {name}: a CUDA tensor of rank 2"):
        ops.dense(operands["x"], on_the_device(4, 4), operands["out"], residual=operands["residual"])


def test_a_parsed_shape_comes_out_of_its_constructor(monkeypatch):
    """All fields, in the constructor's hands: what it does not know is an error and not an attribute that is missing later."""
    names = [f.name for f in dataclasses.fields(PagedAttentionShape)]
    values = dict(zip(names, range(1, len(names) + 1)))
    assert vars(PagedAttentionShape(*values.values())) == vars(PagedAttentionShape(**values)) == values
    required = {f.name: 1 for f in dataclasses.fields(PagedAttentionShape) if f.default is dataclasses.MISSING}
    assert vars(PagedAttentionShape(**required)) == {f.name: 1 if f.default is dataclasses.MISSING else f.default for f in dataclasses.fields(PagedAttentionShape)}
    with pytest.raises(TypeError):
        PagedAttentionShape(**values, block_table=1)
    with pytest.raises(dataclasses.FrozenInstanceError):
        PagedAttentionShape(**values).scale = 2.0
    made = []
    original = PagedAttentionShape.__init__
    monkeypatch.setattr(PagedAttentionShape, "__init__", lambda self, *args, **kw: made.append(self) or original(self, *args, **kw))
    i32 = dict(dtype=torch.int32)
    parsed = parse_paged_attention(torch.zeros(4, 8, 16), torch.zeros(5, 2, 2, 16), torch.zeros(5, 2, 2, 16), torch.zeros(2, 6, **i32), torch.zeros(4, **i32), scale=0.25,
                                   sliding_window=3, keep=torch.zeros(4, 4, **i32))
    assert made == [parsed] and parsed == PagedAttentionShape(4, 8, 16, 5, 2, 2, 6, 0.25, 3, 2, 3, False)
