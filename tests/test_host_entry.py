"""The native Python entry points on the host's side: what they take and which Python errors they
raise.  CPU tensors go as far as the library's own checks."""
import pytest
import torch

import relax_b200
from relax_b200 import ops


@pytest.mark.parametrize("group", [32, 32.0, "32", torch.tensor(32)])
def test_integer_arguments_take_what_int_takes(group):
    x, w, s = torch.zeros(1, 64).half(), torch.zeros(16, 8, dtype=torch.int32), torch.zeros(16, 2).half()
    with pytest.raises(relax_b200.RB200Error, match="CUDA device"):
        ops.gemm_fp16_q4f16(x, w, s, group_size=group)


def test_integer_arguments_refuse_the_rest():
    x, w, s = torch.zeros(1, 64).half(), torch.zeros(16, 8, dtype=torch.int32), torch.zeros(16, 2).half()
    with pytest.raises(TypeError):
        ops.gemm_fp16_q4f16(x, w, s, group_size=[32])


def test_bind_refuses_what_a_call_refuses():
    f = relax_b200.get_global_func("relax_b200.gather_columns")
    x = torch.zeros(1, 64).half()
    with pytest.raises(TypeError):
        f.bind(x, [0], x)
    with pytest.raises(KeyError):
        f.bind(x, torch.zeros(64, dtype=torch.complex64), x)
    f.bind(x, None, x)


def test_host_module_is_rebuilt_for_another_torch(tmp_path, monkeypatch):
    from relax_b200 import _host, build
    abi, commands = tmp_path / "torch_host.abi", []

    def run(cmd, **kw):
        commands.append(cmd)
        return type("Result", (), {"returncode": 0})()

    monkeypatch.setattr(build, "_HOST_ABI", str(abi))
    monkeypatch.setattr(build.subprocess, "run", run)
    abi.write_text(build.host_abi())
    build.build_host()
    assert not commands
    abi.write_text(build.host_abi().replace("torch ", "torch 1"))
    build.build_host()
    assert len(commands) == 1 and abi.read_text() == build.host_abi()
    _host.check_abi(_host.native.built_for, build.host_abi())
    with pytest.raises(RuntimeError, match="rebuild"):
        _host.check_abi("torch 1.0", build.host_abi())


@pytest.mark.gpu
def test_out_of_memory():
    x = torch.empty(1, 64, dtype=torch.float16, device="cuda").expand(1 << 30, 64)
    w = torch.empty(1 << 20, 8, dtype=torch.int32, device="cuda")
    with pytest.raises(torch.OutOfMemoryError):
        ops.gemm_fp16_q4f16(x, w, None)
    torch.empty(16, device="cuda")


@pytest.mark.gpu
def test_results_are_filled_under_deterministic_algorithms():
    """Rows of no expert are left as torch.empty made them, which is NaN under deterministic algorithms."""
    w = ops.preprocess_weight_ft(torch.zeros(2, 64, 16, dtype=torch.int8, device="cuda"), False)
    x, s = torch.zeros(40, 64, device="cuda").half(), torch.ones(2, 16, device="cuda").half()
    indptr = torch.tensor([3, 5], device="cuda")
    torch.use_deterministic_algorithms(True)
    try:
        for rows in (20, 40):
            out = ops.moe_gemm_ft(x[:rows], w, s, indptr)
            assert torch.isfinite(out[:5]).all() and torch.isnan(out[5:]).all()
    finally:
        torch.use_deterministic_algorithms(False)
