"""Which calls the native front of the operators takes and which it leaves to the dispatcher, and that it
needs no care from threads with streams of their own."""
import pytest
import torch

import natten_b200 as nb
import natten_b200._lib as L

pytestmark = pytest.mark.gpu


def _taken(q):
    return nb.functional._native.na(2, q, q, q, 3, None, None, None, None, None, None, False) is not None


def test_calls_that_the_native_front_leaves_alone():
    """Function transforms, modes, subclasses, dual numbers and lazy views need the dispatcher."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    class FunctionMode(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class DispatchMode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Subclass(torch.Tensor):
        pass

    q = torch.randn(2, 9, 9, 2, 64, device="cuda").half()
    assert _taken(q) and _taken(q.clone().requires_grad_()) and _taken(torch.nn.Parameter(q))
    seen = []

    def record(x):
        seen.append(_taken(x))
        return x.float().sum()

    torch.func.vmap(record)(q[None])
    torch.func.grad(record)(q)
    torch.func.functionalize(record)(q)
    torch.func.jvp(record, (q,), (q,))
    with torch.autograd.forward_ad.dual_level():
        record(torch.autograd.forward_ad.make_dual(q, q))
    with FunctionMode():
        record(q)
    with DispatchMode():
        record(q)
    record(torch._neg_view(q))
    seen.append(_taken(q.as_subclass(Subclass)))
    with FakeTensorMode() as mode:
        seen.append(_taken(mode.from_tensor(q)))
    torch.jit.trace(record, (q,), check_trace=False)
    assert seen == [False] * 11
    assert not _taken(q.cpu()) and not _taken(q.to_sparse()) and _taken(q)
    with torch.inference_mode():
        assert torch.equal(nb.na2d(q, q, q, 3), nb.na2d(q.clone(), q, q, 3))


def test_threads_with_streams_of_their_own():
    """Several threads, each on its stream, forward and backward of their own sizes: the same bits as one
    after the other."""
    import threading
    torch.manual_seed(89)
    calls = []
    for i in range(6):
        D, dtype = (64, 128, 32)[i % 3], (torch.bfloat16, torch.float16, torch.float32)[i // 2]
        shape = (40 + i,) if i % 2 else (11 + i, 17)
        leaves = [torch.randn(2, *shape, 2, D, device="cuda").to(dtype).requires_grad_() for _ in range(3)]
        fn = (lambda a: nb.attention(*a, is_causal=True)) if i % 2 else (lambda a: nb.na2d(*a, 5))
        calls.append((fn, leaves, torch.randn_like(leaves[0])))

    def run(call):
        fn, leaves, d_out = call
        out = fn(leaves)
        return [out, *torch.autograd.grad(out, leaves, d_out)]

    want = [run(c) for c in calls]
    torch.cuda.synchronize()
    failed = []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(25):
                    got = run(calls[i])
                torch.cuda.current_stream().synchronize()
                if not all(torch.equal(a, b) for a, b in zip(got, want[i])):
                    failed.append(i)
        except Exception as e:
            failed.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed and L.device_status() == 0
