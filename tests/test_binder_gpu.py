"""The native call path of ``run`` / ``launch`` (csrc/host/binder.cpp) beside the Python one: same results, same errors,
same record.  The first call of a shape is bound in Python, later ones natively."""
import threading

import pytest
import torch

import intent_b200 as ib
from intent_b200.runtime import native

pytestmark = pytest.mark.gpu


def _gemm(device, M=64, K=256, N=128, seed=0):
    g = torch.Generator().manual_seed(seed)
    a = torch.randint(-127, 128, (M, K), generator=g, dtype=torch.int8)
    b = torch.randint(-127, 128, (K, N), generator=g, dtype=torch.int8)
    bias = torch.randint(-9, 9, (N,), generator=g, dtype=torch.int32)
    expected = (a.double() @ b.double()).to(torch.int32) + bias
    return [t.to(device) for t in (a, b, bias)], expected


def test_results_shapes_streams_and_record(cuda_device):
    artifact = ib.compile(ib.programs.gemm_i8, target=ib.B200Target(0))
    for M in (64, 80, 64, 1, 80):                      # plans of several shapes side by side
        inputs, expected = _gemm(cuda_device, M=M, seed=M)
        for _ in range(2):
            assert torch.equal(artifact.run(*inputs).cpu(), expected)
    assert artifact.runtime.binder.last() is not None
    inputs, expected = _gemm(cuda_device, M=80, seed=80)
    launches = native.launch_count()
    out = artifact.run(*inputs)
    assert native.launch_count() == launches + 1 and out.dtype == torch.int32
    seen = artifact.observation
    assert seen.status == 0 and seen.stage == "launched" and seen.arguments[0] == ("a", (80, 256), (256, 1))
    assert seen.kernel.startswith("i8_gemm_kernel") and artifact.observation is seen
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        other = artifact.run(*inputs)
    side.synchronize()
    assert torch.equal(other.cpu(), expected)
    buffer = torch.empty_like(out)
    for _ in range(2):
        artifact.launch(*inputs, buffer)
    assert torch.equal(buffer.cpu(), expected)


def test_workspace_follows_the_stream_and_the_switches(cuda_device):
    artifact = ib.compile(ib.programs.weight_only_int4_matmul, target=ib.B200Target(0),
                          constexprs={"GROUP_SIZE": 128, "ZERO_POINT": 8})
    x, p, s = (t.to(cuda_device) for t in ib.workloads.w4a16_inputs(1, 1024, 512, dtype=torch.float16, seed=1))
    expected = artifact.run(x, p, s)
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    outs = []
    for stream in streams + streams:
        with torch.cuda.stream(stream):
            outs.append(artifact.run(x, p, s))
    torch.cuda.synchronize()
    assert all(torch.equal(o, expected) for o in outs) and len(artifact.runtime._stream_workspaces) == 4
    library = native.library()
    try:
        assert library.intent_b200_w4a16_gemv_warps(16) == 0     # another plan of the same shapes
        out = artifact.run(x, p, s)
        assert artifact.observation.threads == 512
        artifact.run(x, p, s)
    finally:
        library.intent_b200_w4a16_gemv_warps(0)
    assert artifact.observation.threads == 512
    artifact.run(x, p, s)
    assert artifact.observation.threads == 1024
    assert torch.allclose(out.float(), expected.float(), rtol=1e-2, atol=1e-2)
    artifact.check()


def test_errors_are_those_of_the_python_path(cuda_device):
    artifact = ib.compile(ib.programs.gemm_i8, target=ib.B200Target(0))
    (a, b, bias), expected = _gemm(cuda_device)
    artifact.run(a, b, bias)
    artifact.run(a, b, bias)
    with pytest.raises(TypeError, match="expected 3 runtime arguments"):
        artifact.run(a, b)
    with pytest.raises(TypeError, match="must be a torch.Tensor"):
        artifact.run(a, b, 3)
    with pytest.raises(TypeError, match="dtype"):
        artifact.run(a, b, bias.long())
    with pytest.raises(ValueError, match="bound to"):
        artifact.run(a.cpu(), b, bias)
    with pytest.raises(ValueError, match="rank"):
        artifact.run(a[0], b, bias)
    with pytest.raises(ValueError, match="violates the declared interface relation"):
        artifact.run(a[:, :128].contiguous(), b, bias)
    with pytest.raises(NotImplementedError, match="contiguous"):
        artifact.run(a.t().contiguous().t(), b, bias)
    shifted = torch.empty(a.numel() + 1, dtype=torch.int8, device=cuda_device)[1:].view(a.shape)
    with pytest.raises(ValueError, match="alignment"):
        artifact.run(shifted, b, bias)
    out = torch.zeros(64, 128, dtype=torch.int32, device=cuda_device)
    artifact.launch(a, b, bias, out)
    overlapping = bias.new_zeros(64 * 128 + 128)
    with pytest.raises(NotImplementedError, match="nonoverlapping"):
        artifact.launch(a, b, overlapping[:128], overlapping[:64 * 128].view(64, 128))
    empty = artifact.run(a[:0], b, bias)
    assert empty.shape == (0, 128) and torch.equal(artifact.run(a, b, bias).cpu(), expected)
    assert torch.equal(artifact.run(torch.nn.Parameter(a, requires_grad=False), b, bias).cpu(), expected)


def test_several_threads(cuda_device):
    artifact = ib.compile(ib.programs.gemm_i8, target=ib.B200Target(0))
    cases = [_gemm(cuda_device, M=16 * (i + 1), seed=i) for i in range(4)]
    failures = []

    def work(index):
        inputs, expected = cases[index]
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(50):
                out = artifact.run(*inputs)
            torch.cuda.current_stream().synchronize()
            if not torch.equal(out.cpu(), expected):
                failures.append(index)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures


def _binder_of(entry, workspaces):
    """A native caller of ``entry`` (a Python function of the slots) with one f32 input and one f32 output of one axis each.
    Nothing is launched: the entry stands where the library's would."""
    import ctypes

    function = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.POINTER(ctypes.c_int64))(entry)
    switches = ctypes.create_string_buffer(4)
    views = ((0, torch.float32, 1, 4), (1, torch.float32, 1, 4))
    slots = 3 * len(views) + (0 if workspaces is None else 2) + 1
    binder = native._binder_type()(ctypes.cast(function, ctypes.c_void_p).value, slots, 0, ctypes.addressof(switches), 4,
                                   workspaces, views, ())
    return binder, (function, switches)


def test_a_workspace_outlives_the_call_that_uses_it(cuda_device):
    """Another thread may replace the stream's workspace while a call is under way without the interpreter lock; the
    call's buffer must not go back to the allocator before it has been launched on."""
    size = 4 << 20
    stream = torch.cuda.current_stream().cuda_stream
    workspaces = {stream: torch.zeros(size, dtype=torch.uint8, device=cuda_device)}
    given_back = []

    def entry(slots):
        before = torch.cuda.memory_allocated()
        workspaces[stream] = None                # as a call that needs a larger one does
        given_back.append(before - torch.cuda.memory_allocated())
        return 0

    binder, keep = _binder_of(entry, workspaces)
    binder.learn((8, 8), size, False, bytes(4))
    x = torch.zeros(8, device=cuda_device)
    before = torch.cuda.memory_allocated()
    out = binder.run((x,))
    assert out.shape == (8,) and given_back == [0]
    del out
    assert torch.cuda.memory_allocated() == before - size      # and it does go back afterwards


def test_other_threads_run_while_an_output_is_allocated(cuda_device):
    """An allocation that reaches the driver takes milliseconds: the interpreter lock is released for it, as torch.empty
    does."""
    import sys
    import time

    counter, at_entry, stop = [0], [], threading.Event()

    def entry(slots):
        at_entry.append(counter[0])
        return 0

    binder, keep = _binder_of(entry, None)
    binder.learn((8, 1 << 31), -1, False, bytes(4))

    def count():
        while not stop.is_set():
            counter[0] += 1
            time.sleep(0)

    x = torch.zeros(8, device=cuda_device)
    interval = sys.getswitchinterval()
    thread = threading.Thread(target=count)
    progress = []
    try:
        sys.setswitchinterval(30.0)             # the other thread only gets what is given up
        thread.start()
        for _ in range(5):
            torch.cuda.empty_cache()
            before = counter[0]
            out = binder.run((x,))              # 8 GiB that no cached block serves
            progress.append(at_entry[-1] - before)
            del out
    finally:
        stop.set()
        sys.setswitchinterval(interval)
        thread.join()
        torch.cuda.empty_cache()
    assert max(progress) > 5, progress          # (the call of the entry itself gives the lock up once)


def test_launch_with_a_workspace_does_not_ask_the_native_path(cuda_device):
    """Such a call owns its workspace, which the native path does not make."""
    artifact = ib.compile(ib.programs.weight_only_int4_matmul, target=ib.B200Target(0),
                          constexprs={"GROUP_SIZE": 128, "ZERO_POINT": 8})
    x, p, s = (t.to(cuda_device) for t in ib.workloads.w4a16_inputs(1, 1024, 512, dtype=torch.float16, seed=1))
    expected = artifact.run(x, p, s)
    assert torch.equal(artifact.run(x, p, s), expected)
    asked = []

    class Watched:
        def __init__(self, binder):
            self.binder = binder

        def __getattr__(self, name):
            asked.append(name)
            return getattr(self.binder, name)

    artifact.runtime.binder = Watched(artifact.runtime.binder)
    out = torch.empty_like(expected)
    artifact.launch(x, p, s, out)
    assert torch.equal(out, expected) and not {"launch", "start", "learn"} & set(asked), asked
    # nor does a call of tensors that the native path never takes teach it anything
    class Subclass(torch.Tensor):
        pass

    asked.clear()
    assert torch.equal(artifact.run(x.as_subclass(Subclass), p, s), expected)
    assert not {"start", "learn"} & set(asked), asked
