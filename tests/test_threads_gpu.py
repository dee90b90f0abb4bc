"""The layers' native calls from several host threads and on streams other than the default one."""
import threading
import time

import pytest
import torch

from oracle import inputs

pytestmark = pytest.mark.gpu
KINDS = ["latent", "fp8", "moe", "block"]


def _module(kind, seed):
    from swamla_b200.block import NormedResidualFFN
    from swamla_b200.layer import create_moe_layer
    w = inputs.WORKLOADS["tiny_moe_ragged" if kind == "moe" else "tiny_fp8" if kind == "fp8" else "tiny_ragged"]
    cfg = w.config()
    cfg.moe_fp8 = kind == "fp8"
    torch.manual_seed(seed)
    with torch.device("cuda:0"):
        m = create_moe_layer(cfg).to(torch.bfloat16)
        if kind == "block":
            m = NormedResidualFFN(m, w.D)
        xs = [torch.randn(2, t, w.D, dtype=torch.float32 if kind == "block" else torch.bfloat16) for t in (3, 61, 190, 700)]
    return m.train(), xs


def _steps(m, xs, turns):
    """A forward and backward per input, and an evaluation; everything that comes out."""
    layer = getattr(m, "ffn", m)
    out = []
    for _ in range(turns):
        for x in xs:
            xg = x.clone().requires_grad_(True)
            m.zero_grad(set_to_none=True)
            y = m(xg)
            (y.float().square().mean() + layer.get_aux_loss()).backward()
            out += [y.detach(), xg.grad, *[p.grad for p in m.parameters()]]
            layer.router.update_bias_from_last_forward()
            out.append(layer.router.expert_bias.clone())
            with torch.no_grad():
                out.append(m.eval()(x))
            m.train()
    return out


@pytest.mark.parametrize("kind", KINDS)
def test_threads_on_their_own_streams_give_the_serial_bits(kind):
    n, turns = 3, 4
    want = [_steps(*_module(kind, i), turns) for i in range(n)]
    torch.cuda.synchronize()
    jobs, got, errors = [_module(kind, i) for i in range(n)], [None] * n, []
    torch.cuda.synchronize()

    def work(i):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                got[i] = _steps(*jobs[i], turns)
            s.synchronize()
        except Exception as e:                                           # pragma: no cover
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(n)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for a, b in zip(want, got):
        assert len(a) == len(b) and all(torch.equal(p, q) for p, q in zip(a, b))


@pytest.mark.parametrize("kind", ["latent", "moe", "block"])
def test_a_launch_that_waits_for_the_queue_lets_other_threads_run(kind):
    """Behind a one-second kernel the queue fills up and a launch blocks until it ends; the interpreter lock must be free."""
    m, xs = _module(kind, 0)
    x, stop, gaps = xs[2], threading.Event(), []
    with torch.no_grad():
        m(x)
    torch.cuda.synchronize()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    t = threading.Thread(target=tick)
    t.start()
    try:
        torch.cuda._sleep(2_000_000_000)                                 # about a second of a kernel that ends by itself
        t0 = time.perf_counter()
        with torch.no_grad():
            for _ in range(400):                                         # ten launches and more each
                m(x)
        blocked = time.perf_counter() - t0
    finally:
        stop.set()
        t.join()
        torch.cuda.synchronize()
    assert blocked > 0.5, "the queue never filled up"
    assert max(gaps) < 0.3 * blocked, (max(gaps), blocked)


def test_a_failure_names_its_device_and_is_reported_once():
    from swamla_b200 import _cabi, _testing
    m, xs = _module("latent", 0)
    sink = {}
    _testing.SINK = sink
    try:
        m(xs[0])
    finally:
        _testing.SINK = None
    torch.cuda.synchronize()
    sink["status"].fill_(101)                # what a kernel writes when its wait gives up
    with pytest.raises(_cabi.LmoeError, match="101 in LatentMoE forward on cuda:0"):
        m.check_status()
    m.check_status()
    m(xs[0])


@pytest.mark.parametrize("kind", ["latent", "fp8", "moe"])
def test_a_backward_leaves_what_the_forward_saved_as_it_is(kind):
    """Another backward of the same graph may read it at the same time; a second one gives the first one's bits."""
    m, xs = _module(kind, 1)
    x = xs[2].clone().requires_grad_(True)
    saved = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: saved.append(t) or t, lambda t: t):
        y = m(x)
    before = [t.clone() for t in saved]
    grads = [torch.autograd.grad(y, [x, *m.parameters()], torch.ones_like(y), retain_graph=True, allow_unused=True) for _ in range(2)]
    assert saved and all(torch.equal(a, b) for a, b in zip(saved, before))
    assert all(a is b or torch.equal(a, b) for a, b in zip(*grads))


@pytest.mark.parametrize("kind", ["latent", "fp8", "moe", "block", "backward"])
def test_first_call_of_a_thread(kind):
    """A thread whose first CUDA call is the layer's, with every buffer from PyTorch's cache, has no current context before it."""
    from swamla_b200 import functional
    m, xs = _module("latent" if kind == "backward" else kind, 0)
    x = xs[3].repeat(1, 2, 1)                                           # 2,800 tokens: nothing goes to the side stream first
    args = (*m._arguments(), m.n_activated, 1e-3, False) if kind == "backward" else None
    with torch.no_grad():
        if kind == "backward":
            fwd = functional._host().latent_fwd_raw(x, *args, None, False)
            call = lambda: functional._host().latent_bwd_raw(fwd[0], None, x, *args[:7], fwd[2], fwd[4], *args[8:], False)[0][0]
        else:
            call = lambda: m(x)
        want = call()
        call()                                                         # (its buffers go back to the cache)
    torch.cuda.synchronize()
    got = []

    def work():
        torch.set_grad_enabled(False)
        try:
            got.append(call())
        except Exception as e:                                           # pragma: no cover
            got.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert isinstance(got[0], torch.Tensor), got[0]
    assert torch.equal(got[0], want)


@pytest.mark.parametrize("kind", ["latent", "moe"])
def test_no_stream_that_others_use_becomes_part_of_a_capture(kind):
    """PyTorch hands out 32 pooled streams in turn; work on any of them while a layer is being captured has to run."""
    m, xs = _module(kind, 0)
    x, z = xs[2], torch.zeros(1, device="cuda:0")
    main = torch.cuda.Stream()
    pool = [torch.cuda.Stream() for _ in range(64)]
    with torch.no_grad():
        with torch.cuda.stream(main):
            want = m(x)
        torch.cuda.synchronize()
        others, errors = [s for s in pool if s.cuda_stream != main.cuda_stream], []

        def work():
            torch.set_grad_enabled(False)
            try:
                for s in others:
                    with torch.cuda.stream(s):
                        z.add_(1.0)
                    s.synchronize()
            except Exception as e:
                errors.append(e)

        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=main, capture_error_mode="thread_local"):
            got = m(x)
            t = threading.Thread(target=work)
            t.start()
            t.join()
    assert not errors and z.item() == len(others)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
