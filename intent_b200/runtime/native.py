"""ctypes binding of ``libintent_b200.so``.

The library is loaded once per process under a lock (the reference does the
same for its CPU providers, python/intent/runtime/native_artifact.py:193-213,
258-276).  There is no fallback: a missing library or symbol raises
``CompilationStageError('native_loading', ...)``.
"""
from __future__ import annotations

import ctypes
import os
from pathlib import Path
from threading import Lock

from ..errors import CompilationStageError

_LOCK = Lock()
_LIBRARY: ctypes.CDLL | None = None
_ENTRIES: dict = {}
_SELECTION: ctypes.Array | None = None        # the switches, in the library's own memory
_LIB = Path(__file__).resolve().parent.parent / "lib"
_BINDER = None                                # the Binder type of the host extension; False: not built
PLAIN: frozenset = frozenset()                # the tensor types that a native caller takes
_PACKED: dict = {}                            # entry name -> (address, slots) of its packed form; None: it has none

_CARRIERS = {"ptr": ctypes.c_void_p, "bool": ctypes.c_bool, "i8": ctypes.c_int8, "i16": ctypes.c_int16,
             "i32": ctypes.c_int32, "i64": ctypes.c_int64, "f32": ctypes.c_float, "f64": ctypes.c_double}


def library_path() -> Path:
    override = os.environ.get("INTENT_B200_LIB")
    if override:
        return Path(override)
    return Path(__file__).resolve().parent.parent / "lib" / "libintent_b200.so"


def library() -> ctypes.CDLL:
    global _LIBRARY
    with _LOCK:
        if _LIBRARY is None:
            path = library_path()
            if not path.exists():
                raise CompilationStageError(
                    "native_loading",
                    f"{path} is missing; build it with `python -m intent_b200.build` "
                    "(there is no CPU or eager fallback)")
            try:
                _LIBRARY = ctypes.CDLL(str(path))
            except OSError as error:
                raise CompilationStageError("native_loading", f"cannot load {path}: {error}") from error
            _LIBRARY.intent_b200_version.restype = ctypes.c_char_p
            _LIBRARY.intent_b200_status_string.restype = ctypes.c_char_p
            _LIBRARY.intent_b200_status_string.argtypes = [ctypes.c_int]
            _LIBRARY.intent_b200_launch_count.restype = ctypes.c_int64
        return _LIBRARY


def entry(name: str, carriers: tuple):
    """Bind one exported entry; ``carriers`` names the slot types in order
    (without the trailing stream pointer, which is always appended)."""
    lib = library()
    key = (name, carriers)
    with _LOCK:
        function = _ENTRIES.get(key)
        if function is None:
            try:
                # (an index makes a function object of its own; the attribute of that name is one object for all,
                # whose argument types a second binding of the symbol would change under this one)
                function = lib[name]
            except AttributeError as error:
                raise CompilationStageError("native_loading", f"{library_path()} does not export {name}") from error
            function.restype = ctypes.c_int
            function.argtypes = [_CARRIERS[c] for c in carriers] + [ctypes.c_void_p]
            _ENTRIES[key] = function
        return function


def selection() -> bytes:
    """A copy of the process-wide switches of the kernel selection (int32 each)."""
    global _SELECTION
    if _SELECTION is None:
        where = library()["intent_b200_selection"]
        where.restype, where.argtypes = ctypes.c_void_p, [ctypes.c_void_p]
        count = ctypes.c_int32()
        address = where(ctypes.byref(count))
        _SELECTION = (ctypes.c_char * (4 * count.value)).from_address(address)
    return _SELECTION.raw


def binder_path() -> Path:
    """Where the host extension for this interpreter and this torch lies: it is compiled against internals of both
    (dispatch keys, the layout of tensor objects), so one that was built for others must not be loaded."""
    import sysconfig

    import torch

    key = (torch.__version__, str(torch.version.git_version)[:8], f"abi{int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           sysconfig.get_config_var("SOABI"))
    return _LIB / ("intent_b200_binder-" + "-".join(key) + ".so")


def _binder_type():
    """The native call path (csrc/host/binder.cpp), or False where it is not built for this interpreter and this torch:
    every call then takes the Python path, which does the same."""
    global _BINDER, PLAIN
    if _BINDER is None:
        from importlib.util import module_from_spec, spec_from_file_location

        import torch         # (the extension links against its libraries)

        PLAIN = frozenset((torch.Tensor, torch.nn.Parameter))

        path = binder_path()
        _BINDER = False
        if path.exists():
            spec = spec_from_file_location("intent_b200_binder", path)
            try:
                module = module_from_spec(spec)
                spec.loader.exec_module(module)
            except ImportError as error:
                raise CompilationStageError("native_loading", f"cannot load {path}: {error}") from error
            _BINDER = module.Binder
        elif any(_LIB.glob("intent_b200_binder*.so")):
            import warnings

            warnings.warn(f"the native call path was built for another torch or Python ({path.name} is not there): calls "
                          "take the Python path; `python -m intent_b200.build` builds it", RuntimeWarning, stacklevel=2)
    return _BINDER


def binder(entry_name: str, device: int, views: tuple, constants: tuple, workspaces: dict | None):
    """A native caller of one entry: ``views`` are (access, torch dtype, rank, alignment) in declaration order.
    None where the entry has no packed form."""
    kind = _binder_type()
    if not kind:
        return None
    packed = _PACKED.get(entry_name, False)
    if packed is False:
        find = library()["intent_b200_packed_call"]
        find.restype, find.argtypes = ctypes.c_void_p, [ctypes.c_char_p, ctypes.c_void_p]
        slots = ctypes.c_int32()
        address = find(entry_name.encode(), ctypes.byref(slots))
        packed = _PACKED[entry_name] = (address, slots.value) if address and slots.value <= 63 else None
    if packed is None or len(views) > 16 or any(not 1 <= v[2] <= 3 for v in views):
        return None
    if sum(1 + 2 * v[2] for v in views) + len(constants) + (0 if workspaces is None else 2) + 1 != packed[1]:
        return None          # not this entry's parameters
    size = len(selection())
    return kind(*packed, device, ctypes.addressof(_SELECTION), size, workspaces, views, constants)


def status_string(status: int) -> str:
    return library().intent_b200_status_string(int(status)).decode()


def launch_count() -> int:
    return int(library().intent_b200_launch_count())


def version() -> str:
    return library().intent_b200_version().decode()


def check(status: int, entry_name: str, observation=None) -> None:
    if status != 0:
        raise CompilationStageError("provider_invocation",
                                    f"{entry_name} returned status {status}: {status_string(status)}",
                                    observation=observation, status=status)


def set_gemv_launch_overlap(enabled: bool) -> None:
    """Process-wide switch of the bandwidth kernel's programmatic dependent launch: a launch may
    request its packed weights while the previous kernel on the stream is still running.  Only
    valid when the weights are not written by the kernel launched immediately before, nor by one ahead of a row of
    W4A16 calls that come before (static model weights in a decode loop)."""
    check(library().intent_b200_w4a16_gemv_overlap(1 if enabled else 0), "intent_b200_w4a16_gemv_overlap")
