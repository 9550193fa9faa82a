"""A source that changes while the compiler runs leaves a stale object, which the next build makes again; the operators in C++ are made
again with the header whose entry points they call, and not left behind where that fails."""
from shuffle_exchange_b200.native import build


def test_source_edited_during_its_compilation_is_compiled_again(tmp_path, monkeypatch):
    csrc, out = tmp_path / "csrc", tmp_path / "out"
    for d in (csrc, out, tmp_path / "include"):
        d.mkdir()
    src = csrc / "a.cu"
    src.write_text("first")
    monkeypatch.setattr(build, "ROOT", tmp_path)
    monkeypatch.setattr(build, "CSRC", csrc)
    monkeypatch.setattr(build, "OUT_DIR", out)
    monkeypatch.setattr(build, "OBJ_DIR", tmp_path / "obj")
    monkeypatch.setattr(build, "_nvcc", lambda: "nvcc")
    compiled, edit = [], ["second"]

    def run(cmd):
        if "-c" in cmd:
            compiled.append(src.read_text())
            (tmp_path / "obj" / "a.o").write_text("object")
            if edit:
                src.write_text(edit.pop())
        return ""
    monkeypatch.setattr(build, "_run", run)
    for _ in range(3):
        build.build_cuda()
        (out / "libsxb200.so").write_text("library")
    assert compiled == ["first", "second"]


def test_operators_follow_their_header_and_do_not_outlive_a_failed_build(tmp_path, monkeypatch):
    out, header = tmp_path / "out", tmp_path / "include" / "sxb200.h"
    for d in (out, tmp_path / "csrc" / "torch", header.parent):
        d.mkdir(parents=True)
    (tmp_path / "csrc" / "torch" / "native_ops.cpp").write_text("source")
    header.write_text("int sxb_f(int);")
    monkeypatch.setattr(build, "ROOT", tmp_path)
    monkeypatch.setattr(build, "CSRC", tmp_path / "csrc")
    monkeypatch.setattr(build, "OUT_DIR", out)
    monkeypatch.setattr(build, "OBJ_DIR", tmp_path / "obj")
    monkeypatch.setattr(build, "_nvcc", lambda: "/usr/local/cuda/bin/nvcc")
    for other in ("build_cuda", "build_host"):
        monkeypatch.setattr(build, other, lambda *a: None)
    compiled, broken = [], []

    def run(cmd):
        target = out / "_sxb_ops.so" if "-shared" in cmd else tmp_path / "obj" / "ops_native_ops.o"
        if "-c" in cmd:
            if broken:
                raise RuntimeError("no such entry point")
            compiled.append(header.read_text())
        target.write_text("built")
        return ""
    monkeypatch.setattr(build, "_run", run)
    build.build_all()
    build.build_all()
    assert len(compiled) == 1 and (out / "_sxb_ops.so").exists()
    header.write_text("int sxb_f(long);")
    broken.append(1)
    build.build_all()
    assert len(compiled) == 1 and not (out / "_sxb_ops.so").exists()
    broken.clear()
    build.build_all()
    assert compiled == ["int sxb_f(int);", "int sxb_f(long);"] and (out / "_sxb_ops.so").exists()
