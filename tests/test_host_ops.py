"""The native part of the tensor-level wrappers (csrc/host_ops.cpp): it takes positional arguments from ops.py only, and what does not
fit is an exception, not a crash.  Its results are covered by every test of ops.py on a GPU."""
import subprocess
import sys
import threading
from pathlib import Path

import pytest
import torch

from fp4_post_b200 import cabi, ops


@pytest.fixture(scope="module")
def host():
    from fp4_post_b200.build import build
    build()
    return cabi.host()


def test_arguments_that_do_not_fit_are_type_errors(host):
    x = torch.zeros(16, 16)
    for name in ("quantize", "quantize_dual", "quantize_dual_finish", "rmsnorm_quantize", "col_mean", "gemv", "lowrank_scale", "lowrank_factors", "gemm"):
        f = getattr(host, name)
        with pytest.raises(TypeError):
            f()
        with pytest.raises(TypeError):
            f(*["text"] * 40)
    with pytest.raises(TypeError):
        host.col_mean(x, 0)                        # no stream
    with pytest.raises(TypeError):
        host.col_mean(None, 0, 0)
    with pytest.raises((TypeError, OverflowError)):
        host.col_mean(x, 0, -1)


@pytest.mark.parametrize("no", [None, False, 0, ""])
def test_switches_are_truth_values(host, no):
    x = torch.zeros(16, 8)                         # blocks of 16 do not divide it: refused before anything is launched
    assert host.quantize(x, cabi.DTYPE_F32, no, 0, 0, 0, cabi.SF_MMA, 0, 0, None, 0)[0] == -2
    rc, *tensors = host.quantize_dual(x, cabi.DTYPE_F32, 0, 0, 0, cabi.SF_MMA, 0, 0, None, no, 0)
    assert rc == -2 and tensors[6] is None         # no token sums


def test_every_entry_point_it_knows_is_exported(host):
    assert not host.bind("metis_no_such_entry", 0)
    known = [n for n in cabi.EXPORTS if host.bind(n, cabi.C.cast(getattr(cabi.lib(), n), cabi.C.c_void_p).value)]
    assert "metis_nvfp4_gemm" in known and len(known) == 15


def test_the_c_entry_points_do_without_it(host, monkeypatch, tmp_path):
    for name in ("_lib", "_host", "_host_lib"):
        monkeypatch.setattr(cabi, name, None, raising=False)
    monkeypatch.setattr(cabi, "HOST_PATH", tmp_path / "nothing.so")
    assert cabi.lib().metis_nvfp4_sf_bytes(128, 64, cabi.SF_MMA) > 0
    with pytest.raises(cabi.MetisLibraryError):
        cabi.host()


def test_another_torch_or_python_does_not_load_it(host):
    """A module of another ABI is not found under the name that this one asks for, and build() makes the right one."""
    code = ("import sys, sysconfig, torch\n"
            "{change}\n"
            "from fp4_post_b200 import build, cabi\n"
            "assert not cabi.HOST_PATH.exists(), cabi.HOST_PATH\n"
            "cabi.lib()\n"
            "try:\n    cabi.host()\n"
            "except cabi.MetisLibraryError:\n    print('refused', str(cabi.HOST_PATH) in build._host_command())\n")
    for change in ("torch.__version__ = '0.0.1+other'", "real = sysconfig.get_config_var\nsysconfig.get_config_var = lambda n: 'cpython-000' if n == 'SOABI' else real(n)"):
        out = subprocess.run([sys.executable, "-c", code.format(change=change)], capture_output=True, text=True, cwd=Path(__file__).resolve().parents[1])
        assert out.stdout.split() == ["refused", "True"], out.stderr


def test_rows_of_unusual_strides_get_a_leading_dimension():
    one = torch.zeros(64).as_strided((1, 64), (1, 1))
    assert one.is_contiguous() and ops._rows2d(one).stride(0) >= 64
    wide = torch.zeros(4, 80)[:, :64]
    assert ops._rows2d(wide).stride(0) == 80
    assert ops._rows2d(torch.zeros(64, 4).T).stride(0) == 64


@pytest.mark.gpu
def test_calls_from_several_threads(host):
    x = torch.randn(512, 1024, device="cuda").to(torch.bfloat16)
    want = ops.nvfp4_quantize(x)
    wrong = []

    def work():
        st = torch.cuda.Stream()
        st.wait_stream(torch.cuda.default_stream())
        with torch.cuda.stream(st):
            for _ in range(50):
                q = ops.nvfp4_quantize(x)
                mean = ops.col_mean(x)
                if not (torch.equal(q.codes, want.codes) and torch.equal(q.scales, want.scales) and mean.numel() == 1024):
                    wrong.append(1)
    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not wrong
