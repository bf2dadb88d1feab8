"""What the Python layer refuses before a kernel is launched.  The library is a stand-in that counts calls: nothing here needs a GPU."""
import subprocess
import sys

import pytest
import torch

from tlaloc_b200 import ops


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
