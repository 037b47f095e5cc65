"""CPU: the native host path of the launchers (the splat_host extension) and the state behind it, without a device."""
import importlib.util
import os
import shutil
import subprocess
import sys
import textwrap
import threading
import time

import pytest
import torch

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
            vec._splat_plan = ((0, 0, vec._version, vec._version, vec._version, 8), plan, vec, vec, False, 0)
            module = dict(rspmm_output=x, scale=1.0, path=0, lse=None, plan=plan, nnzs=vec,
                          sTod_linear_transformations=vec, sTod_translations=vec)
            assert {call} is None
        print("alive")
        """)
    assert r.returncode == 0 and "alive" in r.stdout, (r.returncode, r.stderr[-2000:])


class _Stream:
    cuda_stream = 0

    def synchronize(self):
        time.sleep(0.05)


def _on_a_machine_without_gpu(monkeypatch):
    """torch's device calls replaced by ones that work here; synchronising gives the other threads a turn."""
    import contextlib
    zeros = torch.zeros
    monkeypatch.setattr(torch, "zeros", lambda *a, device=None, **k: zeros(*a, **k))
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d=None: _Stream())
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda t: t.clone())


def _from_threads(f, count=4):
    results, failures = [], []

    def go():
        try:
            results.append(f())
        except BaseException as e:
            failures.append(e)
    threads = [threading.Thread(target=go) for _ in range(count)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
    return results


def test_mask_scratch_is_set_up_once(monkeypatch):
    """First calls from several threads: one registers the scratch, the others wait for it."""
    import splat_native as n
    _on_a_machine_without_gpu(monkeypatch)
    registered = []

    class Host:
        set_mask_work = staticmethod(lambda *a: registered.append(a))
        acsr_from_mask = staticmethod(lambda m, h: registered[0])
    monkeypatch.setattr(n, "_host", Host)
    monkeypatch.setattr(n, "_MASK_WORK", {})

    class Mask:
        device = torch.device("cuda", 0)
    got = _from_threads(lambda: n.acsr_from_mask(Mask, 16))
    assert len(registered) == 1 and got == [registered[0]] * 4


def test_status_word_is_set_up_once(monkeypatch):
    import splat_native as n
    _on_a_machine_without_gpu(monkeypatch)
    mirrors = []

    class Host:
        set_status = staticmethod(lambda *a: None)

    class Lib:
        splat_set_status_mirror = staticmethod(lambda *a: mirrors.append(a) or 0)
    monkeypatch.setattr(n, "_host", Host)
    monkeypatch.setattr(n, "_lib", Lib)
    monkeypatch.setattr(n, "_STATUS_WORDS", {})
    monkeypatch.setattr(n, "_STATUS_MIRRORS", {})
    words = _from_threads(lambda: n.status_word(torch.device("cuda", 0)))
    assert len(mirrors) == 1 and all(w is words[0] for w in words)


def test_extension_of_another_torch_is_rebuilt(monkeypatch, tmp_path):
    """An installed torch that changes makes the extension stale, whatever the ages of the files."""
    spec = importlib.util.spec_from_file_location("splat_build", os.path.join(ROOT, "triton-fun_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    note = tmp_path / "built-for"
    shutil.copyfile(build.HOST_BUILT_FOR, note)
    monkeypatch.setattr(build, "HOST_BUILT_FOR", str(note))
    commands = []
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, **k: commands.append(cmd))
    build.build_host()
    assert not commands
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    build.build_host()
    assert len(commands) == 1
    build.build_host()
    assert len(commands) == 1


def test_kernels_wait_through_the_tested_functions_only():
    """The bounded waits that splat_selftest_bounded_wait makes run out are the ones in tc_ptx.cuh: no kernel polls a barrier
    in a loop of its own."""
    csrc = os.path.join(ROOT, "triton-fun_b200", "csrc")
    for name in sorted(os.listdir(csrc)):
        if name != "tc_ptx.cuh":
            with open(os.path.join(csrc, name)) as f:
                assert "mbar_try_wait" not in f.read(), name


def test_choice_of_the_fused_band_kernel(monkeypatch):
    import splat_native as n

    def choice(bh, L, d, most, stride=1, single=0, table=True):      # most: longest row
        return n.band_kernel_choice(bh, L, d, (most, stride, stride, 0, single, L, 0, L - single), table)

    monkeypatch.delenv("SPLAT_B200_BAND_TILES", raising=False)
    # waves of 296 tiles: two, two and a bit, two and a half, three, three and a half, four
    assert [choice(t // 16, 2048, 128, 401) for t in (576, 592, 608, 720, 736, 768, 880, 1024, 1040, 1168, 1184, 1216)] == \
        [1, 4, 1, 1, 1, 4, 4, 1, 4, 4, 4, 4]
    # bands of half the class and more: from four waves; bands that grow to that: from six
    assert [choice(t // 16, 2048, 128, 1024) for t in (592, 768, 1040, 1184)] == [1, 1, 1, 4]
    assert [choice(t // 16, 2048, 128, 2048) for t in (592, 768, 1040, 1184)] == [1, 1, 1, 4]
    assert [choice(t // 16, 2048, 128, 1024, single=1) for t in (768, 1184)] == [1, 4]
    assert [choice(t // 16, 2048, 128, 2048, single=1) for t in (592, 768, 1184, 1760, 1776)] == [1, 1, 1, 1, 4]
    assert [choice(t // 64, 8192, 128, 1024, 8, 8) for t in (768, 1216, 1792)] == [1, 1, 4]
    assert [choice(t // 64, 8192, 128, 256, 32, 32) for t in (640, 768, 1216)] == [1, 4, 4]      # classes of two tiles
    assert [choice(t, 128, 128, 128, single=1) for t in (740, 800, 1184)] == [4, 4, 4]           # ... and of one
    assert choice(512, 32768, 128, 1024) == 4
    assert choice(512, 32768, 128, 1024, table=False) == 1
    assert choice(512, 32768, 64, 1024) == 1
    assert choice(512, 32767, 128, 1024, 2) == 1                  # classes of unequal length
    assert choice(65535, 2147483647, 128, 3) == 1                 # more tiles than a grid has
    assert choice(1, 128, 128, 128) == 1
    assert choice(0, 128, 128, 128) < 0
    for forced, d, stride, expected in (("4", 128, 1, 4), ("4", 64, 1, -6), ("4", 128, 3, -6), ("1", 128, 1, 1), ("2", 128, 1, 2),
                                        ("3", 128, 1, 3), ("3", 64, 1, 2), ("2", 32, 1, 1), ("2", 128, 3, 1), ("7", 128, 1, 1)):
        monkeypatch.setenv("SPLAT_B200_BAND_TILES", forced)
        assert choice(1, 256, d, 31, stride) == expected, (forced, d, stride)
    monkeypatch.setenv("SPLAT_B200_BAND_TILES", "4")
    assert choice(1, 256, 128, 31, table=False) == -6
