"""The launchers as native Python functions: argument counts, refusals and the way of every field into the call."""
import ctypes
import os
import shutil
import subprocess
import sys
import sysconfig

import numpy as np
import pytest
import torch

from raftinfer_b200 import _call, _lib
from raftinfer_b200 import kernels as K

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NAMES = [n for n in dir(_call) if n.startswith("rib200_")]


@pytest.mark.parametrize("name", NAMES)
def test_native_launchers_take_the_declared_arguments_and_refuse_what_ctypes_refused(name):
    call, count = getattr(_call, name), len(_lib.PROTOTYPES[name])
    for wrong in (count - 1, count + 1):
        with pytest.raises(TypeError):
            call(*[None] * wrong)
    floats = [1.5] * count  # no pointer, no size, no shape
    with pytest.raises((AttributeError, ctypes.ArgumentError)):
        call(*floats)


def test_refusals_of_the_library_name_the_argument_that_is_off():
    """One argument or field off at a time: the refusal's code and text are the library's own for that one."""
    good = dict(tokens=2, query_heads=16, kv_heads=4, head_dim=256, max_context_tokens=256, past_tokens=0)
    call = lambda shape, dtype=K.DTYPE_BF16, policy=K.Qwen35AttentionLaunchPolicy(), cache_bytes=1 << 30, stream=16: \
        K.qwen35_causal_attention(16, 16, 16, 16, 16, 16, cache_bytes, None, 0, K.Qwen35AttentionShape(**shape), dtype,
                                  policy, stream)
    attempts = [(lambda f=f, v=v: call({**good, f: v}), code, text) for f, v, code, text in
                [("tokens", 0, K.INVALID_ARGUMENT, "tokens must be positive"),
                 ("query_heads", 15, K.INVALID_ARGUMENT, "query_heads must be a multiple of kv_heads"),
                 ("kv_heads", 0, K.INVALID_ARGUMENT, "kv_heads must be positive"),
                 ("head_dim", 255, K.UNSUPPORTED, "head_dim 256"),
                 ("max_context_tokens", 1, K.INVALID_ARGUMENT, "context exceeds the cache capacity"),
                 ("past_tokens", 255, K.INVALID_ARGUMENT, "context exceeds the cache capacity")]]
    attempts += [(lambda: call(good, dtype=9), K.INVALID_ARGUMENT, "unknown activation dtype"),
                 (lambda: call(good, cache_bytes=16), K.INVALID_ARGUMENT, "KV cache is too small"),
                 (lambda: call(good, stream=None), K.INVALID_ARGUMENT, "stream is null"),
                 (lambda: call(good, policy=K.Qwen35AttentionLaunchPolicy(7, 1, 1)), K.INVALID_ARGUMENT,
                  "unknown attention implementation"),
                 (lambda: call(good, policy=K.Qwen35AttentionLaunchPolicy(1, 1, 9)), K.INVALID_ARGUMENT,
                  "unknown KV cache layout")]
    for attempt, code, text in attempts:
        with pytest.raises(K.Qwen35PrimitiveError, match=text) as refusal:
            attempt()
        assert refusal.value.code == code
    delta = dict(tokens=2, hidden_size=256, key_heads=1, value_heads=2, key_dim=128, value_dim=128, conv_width=4,
                 epsilon=1.0e-6)
    call = lambda shape, policy=K.GatedDeltaLaunchPolicy(): \
        K.qwen35_gated_delta(16, 16, 16, 16, 16, 16, 16, 16, 16, 1 << 30, K.GatedDeltaShape(**shape), K.DTYPE_F32,
                             K.DTYPE_F32, 16, policy)
    attempts = [(lambda f=f, v=v: call({**delta, f: v}), text) for f, v, text in
                [("tokens", 0, "tokens must be positive"), ("hidden_size", 255, "must equal hidden_size"),
                 ("key_heads", 3, "value_heads must be a multiple of key_heads"),
                 ("value_heads", 3, "must equal hidden_size"), ("key_dim", 0, "key_dim must be positive"),
                 ("value_dim", 64, "must equal hidden_size"), ("conv_width", 0, "conv_width must be positive"),
                 ("epsilon", -1.0, "epsilon must be finite and non-negative")]]
    attempts += [(lambda p=p: call(delta, p), text) for p, text in
                 [(K.GatedDeltaLaunchPolicy(9, 4, False), "unknown gated-delta schedule"),
                  (K.GatedDeltaLaunchPolicy(0, 3, False), "four warps per block"),
                  (K.GatedDeltaLaunchPolicy(0, 4, True), "transposed boundary state")]]
    for attempt, text in attempts:
        with pytest.raises(K.Qwen35DeltaError, match=text) as refusal:
            attempt()
        assert refusal.value.code == K.INVALID_ARGUMENT


# ---- against ctypes, on stand-ins that record what arrives (cpp/recording_stub.cpp) ----
class Tensor:
    def __init__(self, address):
        self.address = address

    def data_ptr(self):
        return self.address


class Stream:
    cuda_stream = 0x5EED_0000_0001


@pytest.fixture(scope="module")
def recorder(tmp_path_factory):
    """call(name, arguments, native) -> the bytes that arrive, or the exception's type and text."""
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    library = str(tmp_path_factory.mktemp("stub") / "librecording.so")
    subprocess.run([cxx, "-std=c++17", "-O1", "-fPIC", "-shared", os.path.join(ROOT, "tests", "cpp", "recording_stub.cpp"),
                    "-o", library], check=True)
    stub = ctypes.CDLL(library)
    stub.stub_address.argtypes, stub.stub_address.restype = [ctypes.c_char_p], ctypes.c_void_p
    stub.stub_record.argtypes, stub.stub_record.restype = [ctypes.c_void_p, ctypes.c_size_t], ctypes.c_size_t
    buffer = ctypes.create_string_buffer(4096)
    address = lambda name: stub.stub_address(name.encode())

    def through_ctypes(name, *arguments):
        function = ctypes.CFUNCTYPE(_lib.Status, *_lib.PROTOTYPES[name])(address(name))
        assert function(*K._ctypes_arguments(name, arguments)).code == 0

    def call(name, arguments, native):
        try:
            getattr(_call, name)(*arguments) if native else through_ctypes(name, *arguments)
        except Exception as error:  # noqa: BLE001 - the type and the text are what is compared
            assert stub.stub_record(buffer, len(buffer)) == 0
            return type(error), str(error)
        arrived = stub.stub_record(buffer, len(buffer))
        return buffer.raw[:arrived]

    _call.bind(address, through_ctypes, K.Qwen35PrimitiveError, K.Qwen35DeltaError)
    yield call
    _call.bind(lambda name: ctypes.cast(getattr(_lib.lib, name), ctypes.c_void_p).value, K._through_ctypes,
               K.Qwen35PrimitiveError, K.Qwen35DeltaError)


def plain_arguments(name):
    """A distinct value in every argument and in every field of a shape, a plan or a policy."""
    count = iter(range(1, 1000))
    size, byte = lambda: (1 << 40) + next(count), lambda: next(count)
    make = {
        _lib.AttentionShape: lambda: K.Qwen35AttentionShape(*[size() for _ in range(6)]),
        _lib.QkNormRopeShape: lambda: K.QkNormRopeShape(*[size() for _ in range(5)], next(count) + 0.125),
        _lib.OnlineDecodePlan: lambda: K.Qwen35OnlineDecodePlan(byte(), *[size() for _ in range(4)]),
        _lib.GatedDeltaShape: lambda: K.GatedDeltaShape(*[size() for _ in range(7)], next(count) + 0.25),
        _lib.AttentionLaunchPolicy: lambda: K.Qwen35AttentionLaunchPolicy(byte(), byte(), byte()),
        _lib.GatedDeltaLaunchPolicy: lambda: K.GatedDeltaLaunchPolicy(byte(), 70000 + byte(), True),
        _lib.vp: lambda: Tensor((1 << 44) + 16 * next(count)), _lib.sz: size,
        ctypes.c_int32: lambda: -next(count), ctypes.c_uint8: byte, ctypes.c_float: lambda: next(count) + 0.5,
    }
    types = _lib.PROTOTYPES[name]
    arguments = [make[getattr(t, "_type_", None) if hasattr(t, "_type_") and not isinstance(t._type_, str) else t]()
                 for t in types]
    arguments[len(types) - (2 if name == "rib200_qk_norm_rope" else 1)] = Stream()
    return arguments


@pytest.mark.parametrize("name", NAMES)
def test_every_argument_arrives_as_through_ctypes(name, recorder):
    arguments = plain_arguments(name)
    native = recorder(name, arguments, True)
    assert isinstance(native, bytes) and native == recorder(name, arguments, False)
    seen = {native}
    for i, x in enumerate(arguments):  # addresses, none and numbers at the ends of their ranges in place of each
        for other in [None, 0, 7, True, -1, 2 ** 31, 2 ** 63, 2 ** 64 - 1]:
            changed = arguments[:i] + [other] + arguments[i + 1:]
            assert recorder(name, changed, True) == recorder(name, changed, False), (i, other)
        if isinstance(x, (Tensor, Stream)):
            seen.add(recorder(name, arguments[:i] + [64 * i + 5] + arguments[i + 1:], True))
    assert len(seen) == 1 + sum(isinstance(x, (Tensor, Stream)) for x in arguments)


@pytest.mark.parametrize("name", NAMES)
def test_what_ctypes_accepts_is_accepted_and_what_it_refuses_refused_alike(name, recorder):
    """Integers of numpy and torch, ctypes numbers, floats, strings: in every argument and in every field of a shape."""
    others = [np.int64(9), np.uint8(9), np.float32(1.5), torch.tensor(9), torch.tensor(1.5), torch.zeros(2), 1.5,
              float("nan"), "9", b"9", object(), ctypes.c_size_t(9), ctypes.c_int32(9), ctypes.c_float(1.5), [9]]
    arguments = plain_arguments(name)
    accepted = 0
    for i, x in enumerate(arguments):
        for other in others:
            candidates = [other]
            if hasattr(x, "c"):  # in each field of a shape, a plan or a policy
                candidates += [type(x)(**{**vars(x), field: other}) for field in vars(x)]
            for candidate in candidates:
                changed = arguments[:i] + [candidate] + arguments[i + 1:]
                native, reference = recorder(name, changed, True), recorder(name, changed, False)
                text = lambda r: r if isinstance(r, bytes) else (r[0], r[1].split(" at 0x")[0])
                assert text(native) == text(reference), (i, candidate)
                accepted += isinstance(native, bytes)
    assert accepted > 0


# ---- the built file ----
def test_the_native_functions_are_of_this_interpreter_and_say_how_to_be_built(tmp_path):
    """The file carries the interpreter's ABI tag; where it is missing the import names the way to build it, and a make
    without Python's headers still gives the library."""
    assert _call.__file__.endswith(sysconfig.get_config_var("EXT_SUFFIX"))
    package = os.path.join(ROOT, "raftinfer_b200")
    (tmp_path / "raftinfer_b200").mkdir()
    for name in ("__init__.py", "_lib.py", "kernels.py", "librib200.so"):
        os.symlink(os.path.join(package, name), tmp_path / "raftinfer_b200" / name)
    run = subprocess.run([sys.executable, "-c", "import raftinfer_b200.kernels"], cwd=tmp_path, capture_output=True,
                         text=True, env={**os.environ, "PYTHONPATH": ""})
    assert run.returncode != 0 and "built for another interpreter" in run.stderr and "g.build()" in run.stderr
    if shutil.which("make"):
        plan = subprocess.run(["make", "-n", "-C", os.path.join(package, "csrc"), "PYTHON=/nonexistent/python"],
                              capture_output=True, text=True)
        assert plan.returncode == 0 and "binding.cpp" not in plan.stdout
