"""A source that changes while the compiler runs leaves a stale object, which the next build makes again."""
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
