"""ctypes loader of libhipster_b200.so. Fails loudly when the CUDA library is missing: there is no CPU fallback."""
import ctypes
import os
import re

HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.environ.get("HIPSTER_B200_LIB") or os.path.join(HERE, "libhipster_b200.so")
HEADER = os.path.join(HERE, "..", "include", "hipster_b200.h")

_lib = _hot = None
# the calls whose latency counts, with their argument types (p pointer, i int, f float), so that integers pass without a wrapper object
_TYPES = {"p": ctypes.c_void_p, "i": ctypes.c_int, "f": ctypes.c_float}
_HOT = {"hp_quantize_x_q8": "piiippp", "hp_gemv_q4k_q8": "ppppiiiip", "hp_argmax": "piiipppp", "hp_accept_greedy": "ppipp", "hp_attn_decode": "piiiiiipppppipppfpp"}


class HipsterError(RuntimeError):
    """Raised for every non-zero status of the C ABI (the reference throws std::runtime_error, qwen35.cpp:10)."""

    def __init__(self, code, msg):
        super().__init__(f"hipster_b200 error {code}: {msg}")
        self.code = code


def declared_symbols():
    """Names of the functions declared in include/hipster_b200.h."""
    text = open(HEADER).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(hp_[a-z0-9_]+)\s*\(", text)))


def lib():
    global _lib
    if _lib is None:
        if not os.path.exists(LIB_PATH):
            raise HipsterError(-1, f"{LIB_PATH} is missing: build it with `python -m hipster_b200.build` (needs nvcc); no fallback path exists")
        _lib = ctypes.CDLL(LIB_PATH)
        _lib.hp_last_error.restype = ctypes.c_char_p
        for name in ("hp_xq8_q_bytes", "hp_xq8_sc_bytes", "hp_argmax_scratch_bytes", "hp_attn_workspace_bytes"):
            getattr(_lib, name).restype = ctypes.c_size_t
    return _lib


def hot():
    """The calls of _HOT with integers (None: absent) for every argument. They go through csrc/pycalls.c, bound to the library that is loaded here;
    where that module is not there (a package with the library alone, another interpreter than the one it was built for), through ctypes, a
    microsecond slower each, on function objects of this package's own: those of lib() take whatever ctypes objects a caller passes."""
    global _hot
    if _hot is None:
        L = lib()
        try:
            from . import _calls as calls
        except ImportError:
            calls = ctypes.CDLL(LIB_PATH)
            for name, types in _HOT.items():
                getattr(calls, name).argtypes = [_TYPES[t] for t in types]
        else:
            for name in _HOT:
                calls.bind(name, ctypes.cast(getattr(L, name), ctypes.c_void_p).value)
        _hot = calls
    return _hot


def check(code):
    if code != 0:
        raise HipsterError(code, lib().hp_last_error().decode())
    return code


def ptr(t):
    """Device (or host) pointer of a torch tensor / numpy array as c_void_p; None -> NULL."""
    if t is None:
        return ctypes.c_void_p(0)
    try:
        return ctypes.c_void_p(t.data_ptr())
    except AttributeError:
        return ctypes.c_void_p(t.ctypes.data)
