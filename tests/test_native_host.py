"""CPU: the native host path of the launchers (the splat_host extension) and the state behind it, without a device."""
import subprocess
import sys
import textwrap

import pytest

from conftest import ROOT, SPLAT_DIR


def run_python(code):
    head = f"import sys; sys.path[:0] = [{ROOT!r}, {SPLAT_DIR!r}]\nimport torch\n"
    return subprocess.run([sys.executable, "-c", head + textwrap.dedent(code)], capture_output=True, text=True, timeout=300)


@pytest.mark.parametrize("call", ["n._host.softmax(x, x, vec, 8, 1.0)",
                                  "n._host.sddmm(x, x.transpose(2, 3), x, vec, vec, vec, 8, 0)",
                                  "n._host.spmm(x, x, x, vec, vec, vec, 8, 0)",
                                  "n._host.module_forward(module, [x, x.transpose(2, 3), x])"])
def test_operands_without_data_end_no_process(call):
    """Tensors that torch refuses to give the data (or even the strides) of: no answer or a Python exception, not the
    end of the process."""
    r = run_python(f"""
        import ctypes
        import splat_native as n
        from torch._subclasses.fake_tensor import FakeTensorMode
        words = (ctypes.c_int32 * 2)()
        n._host.set_status(0, ctypes.addressof(words), ctypes.addressof(words) + 4)
        with FakeTensorMode(allow_non_fake_inputs=True):
            x, vec = torch.empty(1, 1, 8, 8, device="cuda:0"), torch.empty(8, device="cuda:0")
            plan = (8, 1, 1, 0, 0, 8, 0, 8)
            vec._splat_plan = ((0, 0, vec._version, vec._version, vec._version, 8), plan, vec, vec, None, 0)
            module = dict(rspmm_output=x, scale=1.0, path=0, lse=None, plan=plan, nnzs=vec,
                          sTod_linear_transformations=vec, sTod_translations=vec)
            assert {call} is None
        print("alive")
        """)
    assert r.returncode == 0 and "alive" in r.stdout, (r.returncode, r.stderr[-2000:])
