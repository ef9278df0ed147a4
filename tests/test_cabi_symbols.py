"""The C-ABI library loads (no GPU needed) and exports every function that include/mok_b200.h declares."""
import ctypes
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_functions():
    text = open(os.path.join(ROOT, "include", "mok_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(mokb_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_are_exported():
    lib = ctypes.CDLL(os.path.join(ROOT, "mixture-of-kittens_b200", "mok", "libmok_b200.so"))
    names = declared_functions()
    assert len(names) >= 18
    for n in names:
        assert hasattr(lib, n), f"{n} is declared in include/mok_b200.h but not exported"


def test_binding_matches_header():
    from mok import _C, _C_mxfp8
    bound = set(_C.EXPORTED) | set(_C_mxfp8.EXPORTED)
    assert bound <= set(declared_functions()), bound - set(declared_functions())
    missing = set(declared_functions()) - bound
    assert not missing, f"declared but not bound in mok/_C.py: {missing}"


def test_argument_errors_without_a_gpu():
    from mok import _C
    lib = _C.lib
    assert lib.mokb_schedule_scratch_bytes(8, 32) > 8 * 32 * 1024 * 4
    assert lib.mokb_layer_scratch_bytes(1024, 4, 1024) > 0
    rc = lib.mokb_mxfp8_quantize(None, 1, 128, 128, None, None, None, None, None)
    assert rc == -1 and b"null input" in _C._last_error()
    rc = lib.mokb_schedule(None, 1, 512, 2, 4, 2048, 0, None, None, None, None, None, None, None)
    assert rc == -1 and b"null pointer" in _C._last_error()


def test_the_quantising_pull_refuses_rows_that_its_stores_would_leave():
    """Its warps store 32 rows and 32 token columns at a time: checked before anything is launched (the addresses are never read)."""
    from mok import _C
    src = (ctypes.c_uint64 * 1)(4096)
    def call(max_rows, row_begin, row_end, t_rows):
        vp = lambda: ctypes.c_void_p(4096)
        return _C.lib.mokb_dispatch_rows_quant(src, 1, vp(), vp(), None, max_rows, row_begin, row_end, 1, 256, None, None, vp(), vp(), vp(), vp(),
                                               t_rows, 0, None, None, 0, 0, None, None)
    for args, why in (((100, 0, 128, 128), b"multiples of 128"), ((256, 0, 100, 256), b"multiples of 128"), ((-128, 0, 128, 128), b"multiples of 128"),
                      ((256, 0, 256, 128), b"do not fit"), ((512, 128, 512, 256), b"do not fit")):
        assert call(*args) == -1 and why in _C._last_error(), args
    assert call(0, 0, 0, 128) == 0 and call(256, 256, 512, 256) == 0      # no rows: nothing to do
