"""CPU: what build.py decides to build (no compiler runs): the library without torch, the torch module on
top of it where torch is installed, and that again when torch or Python changes."""
import importlib.util
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def _script(tmp_path, monkeypatch):
    spec = importlib.util.spec_from_file_location("package_build", ROOT / "ascend-fft_b200" / "build.py")
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    made = []

    def compile_one(cmd):
        out = Path(cmd[cmd.index("-o") + 1])
        out.write_text("")
        made.append(out.name)
        return ""

    for name, value in (("BUILD", tmp_path / "_build"), ("LIBDIR", tmp_path / "lib"),
                        ("LIB", tmp_path / "lib" / "libbfly_b200.so"), ("TORCH_LIB", tmp_path / "lib" / "_torch_ops.so"),
                        ("compile_one", compile_one), ("nvcc", lambda: "/usr/local/cuda/bin/nvcc")):
        monkeypatch.setattr(b, name, value)
    return b, made


def test_library_needs_no_torch(tmp_path, monkeypatch):
    b, made = _script(tmp_path, monkeypatch)
    monkeypatch.setattr(b, "torch_abi", lambda: None)
    monkeypatch.setattr(b, "torch_cmd", None)   # importing torch would fail
    assert b.build() == b.LIB and b.LIB.exists() and not b.TORCH_LIB.exists()
    assert not any("torch" in m for m in made)


def test_module_follows_torch_and_python(tmp_path, monkeypatch):
    b, made = _script(tmp_path, monkeypatch)
    b.build()
    assert b.LIB.exists() and b.TORCH_LIB.exists() and "torch_ops.torch.o" in made
    made.clear()
    b.build()
    assert made == []
    monkeypatch.setattr(b, "torch_abi", lambda: "torch 99.0 another-python")
    b.build()
    assert made == ["torch_ops.torch.o", "_torch_ops.so.tmp"]
    made.clear()
    b.build()
    assert made == []
    b.TORCH_LIB.unlink()
    b.build()
    assert made == ["_torch_ops.so.tmp"]
