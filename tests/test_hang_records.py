"""Every kernel family that can give up a wait is asked, by the benchmark, the serving benchmark and the smoke run alike."""
import ctypes
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _text(*parts):
    with open(os.path.join(ROOT, *parts)) as f:
        return f.read()


def test_all_families_are_known():
    from shuffle_exchange_b200.native import lib
    kinds = {k for p in glob.glob(os.path.join(ROOT, "csrc", "*.cu"))
             for k in re.findall(r"SXB_DEFINE_HANG_ACCESSOR\(sxb_(\w+)_hang_info\)", _text("csrc", p))}
    assert kinds == set(lib.HANG_KINDS)


def test_a_record_of_any_family_is_found(monkeypatch):
    from shuffle_exchange_b200.native import lib

    class Fake:
        def __init__(self, bad):
            self.bad = bad

        def __getattr__(self, name):
            def accessor(out):
                words = ctypes.cast(out, ctypes.POINTER(ctypes.c_uint))
                for i in range(8):
                    words[i] = (i + 1) * (name == f"sxb_{self.bad}_hang_info")
                return 0
            return accessor

    monkeypatch.setattr(lib.torch.cuda, "synchronize", lambda: None)
    for bad in lib.HANG_KINDS:
        monkeypatch.setattr(lib, "load", lambda bad=bad: Fake(bad))
        assert lib.hang_any() == {bad: {"tag": 2, "block": (3, 4, 5), "thread": 6, "parity": 7, "aux": 8}}
    monkeypatch.setattr(lib, "load", lambda: Fake("none"))
    assert lib.hang_any() is None


def test_benchmarks_and_smoke_ask_all_of_them():
    bench, entry = _text("bench.py"), _text("__graft_entry__.py")
    assert "hang_info(" not in bench and bench.count("hang_any()") == 3       # behind the warm-up, at the end, behind serving
    assert "hang_info(" not in entry and "assert lib.hang_any() is None" in entry
