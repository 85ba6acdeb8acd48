"""The compiled host side of a launch: argument kinds against the launchers' own parameters, conversions, errors (no GPU)."""

import ctypes
import os
import re

import pytest
import torch

from freetoken_b200.csrc import build, ops


def _declared():
    """``(library, launcher, kinds)`` as the ops' faces name them."""
    with open(os.path.join(build.HERE, "ops.py")) as f:
        return re.findall(r'_fn\("(\w+)",\s*"(\w+)",\s*"([^"]+)"', f.read())


@pytest.mark.parametrize("lib,name,kinds", _declared(), ids=[f"{n}-{i}" for i, (_, n, _) in enumerate(_declared())])
def test_kinds_are_the_launchers_parameters(lib, name, kinds):
    with open(os.path.join(build.HERE, build.LIBRARIES[lib])) as f:
        source = f.read()
    parameters = re.search(r"\bint %s\(([^)]*)\)" % name, source).group(1).split(",")
    assert parameters.pop().split() == ["cudaStream_t", "stream"]
    kind = lambda p: "p" if "*" in p else "q" if "long long" in p else "f" if p.split()[0] == "float" else "i"
    assert [kind(p) for p in parameters] == kinds.split()
    assert f"FT_PACKED({name})" in source


@pytest.fixture
def host():
    module = build.load_host()
    module.setup(torch.Tensor, lambda: 3, lambda device: 1000 + device, ops.KernelError, ops._ERRORS)
    yield module
    module.setup(torch.Tensor, getattr(torch._C, "_cuda_getDevice", lambda: 0),
                 getattr(torch._C, "_cuda_getCurrentRawStream", lambda d: 0), ops.KernelError, ops._ERRORS)


def _launcher(host, kinds, code=0, kernels=1):
    """A launcher that notes the words it was given."""
    seen = []

    def packed(words):
        at = (ctypes.c_longlong * (len(kinds.split()) + 1)).from_address(words)
        seen.append(list(at))
        return code
    packed = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p)(packed)
    launcher = host.Launcher(ctypes.cast(packed, ctypes.c_void_p).value, kinds, "ft_thing", kernels)
    launcher_and_owner = (launcher, packed)
    return launcher_and_owner, seen


def test_arguments_arrive(host):
    (f, _owner), seen = _launcher(host, "p p p p i q f i", kernels=2)
    t, buffer = torch.zeros(4), ctypes.create_string_buffer(16)
    before = host.count()
    assert f(t, None, 12345, buffer, -7, 1 << 40, 0.5, True) is None
    words = seen[0]
    assert words[:4] == [t.data_ptr(), 0, 12345, ctypes.addressof(buffer)]
    assert words[4:6] == [-7, 1 << 40] and words[7] == 1
    assert ctypes.c_double.from_buffer(ctypes.c_longlong(words[6])).value == 0.5
    assert words[8] == 1003                                   # the current stream of the current device
    assert host.count() - before == 2


def test_what_is_refused(host):
    (f, _owner), seen = _launcher(host, "p i")
    with pytest.raises(TypeError):
        f(None)
    with pytest.raises(TypeError):
        f(None, 1, 2)
    with pytest.raises(TypeError):
        f(None, 1.5)
    with pytest.raises(TypeError):
        f(object(), 1)
    with pytest.raises(ops.KernelError, match="32 bits"):
        f(None, 1 << 31)
    assert seen == []
    with pytest.raises(ValueError):
        host.Launcher(1, "p x", "ft_thing", 1)
    with pytest.raises(ValueError):
        host.Launcher(1, "p " * 49, "ft_thing", 1)


@pytest.mark.parametrize("code,message", [(-101, "thing: unsupported element type"), (-102, "thing: unsupported shape"),
                                          (9, "thing: CUDA error 9")])
def test_codes_are_kernel_errors(host, code, message):
    (f, _owner), _ = _launcher(host, "i", code=code)
    with pytest.raises(ops.KernelError, match=message):
        f(1)


def test_tensors_are_checked(host):
    with pytest.raises(ops.KernelError, match="x must be a CUDA tensor"):
        host.need(torch.zeros(2), "x")

    class OnTheGpu:
        is_cuda, dtype = True, torch.float32

        def is_contiguous(self):
            return False
    t = OnTheGpu()
    assert host.need(t, "x", contiguous=False) is None
    assert host.need(t, "x", torch.float32, False) is None
    with pytest.raises(ops.KernelError, match="x must be torch.bfloat16, is torch.float32"):
        host.need(t, "x", torch.bfloat16)
    with pytest.raises(ops.KernelError, match="x must be contiguous"):
        host.need(t, "x", dtype=torch.float32)
    with pytest.raises(TypeError):
        host.need(t, "x", shape=1)


def test_each_build_of_the_interpreter_has_its_own_module(monkeypatch):
    """A debug or free-threaded interpreter of the same version, or one of another platform, lays objects out otherwise."""
    real = build.sysconfig.get_config_var
    paths = set()
    for abi in ("cpython-312-x86_64-linux-gnu", "cpython-312d-x86_64-linux-gnu", "cpython-312t-x86_64-linux-gnu",
                "cpython-312-aarch64-linux-gnu"):
        monkeypatch.setattr(build.sysconfig, "get_config_var", lambda name, abi=abi: abi if name == "SOABI" else real(name))
        paths.add(build.host_path("/somewhere"))
    assert len(paths) == 4


def test_a_registered_library_without_packed_forms_is_called_too(monkeypatch, tmp_path):
    """A launcher as a library of one's own has it: arguments, then the stream, a code back."""
    import shutil
    import subprocess
    source = tmp_path / "own.c"
    source.write_text("""long long seen[6];
        int ft_own(const void* a, int n, long long m, float f, const void* buffer, void* stream) {
          seen[0] = (long long)a; seen[1] = n; seen[2] = m; seen[3] = (long long)(f * 8);
          seen[4] = (long long)buffer; seen[5] = (long long)stream;
          return n < 0 ? -102 : n > 100 ? 9 : 0; }""")
    subprocess.run([shutil.which("gcc") or "cc", "-shared", "-fPIC", "-o", str(tmp_path / "own.so"), str(source)], check=True)
    library = ctypes.CDLL(str(tmp_path / "own.so"))
    monkeypatch.setattr(build, "load", lambda name: library)
    monkeypatch.setattr(ops, "_bound", {})
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 3, raising=False)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: 1000 + device, raising=False)
    f = ops._fn("own", "ft_own", "p i q f p")
    t, buffer, before = torch.zeros(4), ctypes.create_string_buffer(16), ops.launch_count()
    f(t, 5, 1 << 40, 0.5, buffer)
    assert list((ctypes.c_longlong * 6).in_dll(library, "seen")) == [t.data_ptr(), 5, 1 << 40, 4, ctypes.addressof(buffer), 1003]
    f(None, 5, 1, 0.5, 12345)
    assert ops.launch_count() - before == 2
    with pytest.raises(ops.KernelError, match="own: unsupported shape"):
        f(t, -1, 0, 0.0, None)
    with pytest.raises(ops.KernelError, match="own: CUDA error 9"):
        f(t, 101, 0, 0.0, None)
    with pytest.raises((TypeError, ctypes.ArgumentError)):
        f(t)
