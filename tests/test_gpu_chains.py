"""The chained matcher and the streaming state that is built on it, where they can go wrong: lengths
around a step of 16 positions and a tile of 32 rows, every context length, horizons below it, rows on
chains too long to follow, histories whose step numbers need wide table entries; and the native form
of the differentiable call against the Python one.  All results are exact."""
import numpy as np
import pytest
import torch

from oracle import rosa_oracle as orc
from tests.helpers import nonzero_randn

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _streams(n, heads, bits, seed, alphabet=None, copies=True):
    """Query and key symbols [n, heads] (uint32); the query stream repeats passages of the key's."""
    rng = np.random.default_rng(seed)
    letters = rng.integers(0, 1 << bits, size=alphabet or 1 << min(bits, 16), dtype=np.uint64)
    if alphabet is None and bits <= 16:
        letters = np.arange(1 << bits, dtype=np.uint64)
    q, k = (letters[rng.integers(0, len(letters), size=(n, heads))].astype(np.uint32) for _ in range(2))
    if copies:
        for _ in range(max(1, n // 64)):
            length = int(rng.integers(1, 41))
            if n > 2 * length:
                src, dst = (int(x) for x in rng.integers(0, n - length, size=2))
                q[dst:dst + length] = k[src:src + length]
    return q, k


def _logits(symbols, bits):
    ones = (symbols[..., None] >> np.arange(bits, dtype=np.uint32)) & 1
    return torch.from_numpy(np.where(ones == 1, 0.7, -0.7).astype(np.float32)).to(DEV)


LENGTHS = (1, 15, 16, 17, 31, 33, 129, 256, 511)


@pytest.mark.parametrize("bits,W,alphabet", [
    (1, 300, None), (1, 5, None), (2, 64, None), (3, 2, None), (3, 64, None), (4, 3, None), (5, 32, None),
    (6, 1, None), (7, 16, None), (8, 32, None), (11, 32, None), (12, 32, 40), (16, 20, 300), (32, 32, 60),
    (1, 40, 1), (8, 300, 2), (20, 300, 2)])          # the last three: chains too long to follow
def test_routes_of_packed_sequences_equal_the_oracle(bits, W, alphabet):
    from rosa_soft_b200 import cabi
    H = 3
    cu = np.concatenate([[0], np.cumsum(LENGTHS)])
    q, k = _streams(int(cu[-1]), H, bits, 17 * bits + W, alphabet)
    v = nonzero_randn((int(cu[-1]), 1, 3), 5).to(DEV)
    _, _, _, routes, _ = cabi.hard_forward(_logits(q, bits), _logits(k, bits), v,
                                           torch.from_numpy(cu.astype(np.int32)).to(DEV), W)
    _, want = orc.hard_forward(_logits(q, bits).cpu().numpy(), _logits(k, bits).cpu().numpy(),
                               v.cpu().numpy(), cu, W)
    starts = np.repeat(cu[:-1], LENGTHS)[:, None]
    assert np.array_equal(routes.cpu().numpy(), np.where(want > 0, want + starts, -1))


@pytest.mark.parametrize("T", (2047, 4096, 4113))
@pytest.mark.parametrize("bits,W", [(2, 200), (8, 32), (32, 32)])
def test_long_sequences_of_few_heads_are_indexed_in_pieces(bits, W, T):
    import rosa_soft_b200 as rs
    from rosa_soft_b200 import cabi
    H = 2
    q, k = _streams(T, H, bits, T + bits, None if bits <= 8 else 500)
    pay = np.random.default_rng(3).standard_normal((T, 1, 4)).astype(np.float32)
    want_out, want_end = orc.hard_inference(q, k, pay, np.array([0, T]), W)
    as_int = lambda x: torch.from_numpy(x.view(np.int32))[None].to(DEV)  # noqa: E731
    out, end = rs.rosa_hard_inference(as_int(q), as_int(k), torch.from_numpy(pay)[None].to(DEV),
                                      max_suffix_length=W)
    assert np.array_equal(end[0].cpu().numpy(), want_end)
    assert np.array_equal(out[0].cpu().numpy(), want_out)
    if bits <= 8:
        routes = cabi.hard_forward(_logits(q, bits), _logits(k, bits), torch.from_numpy(pay).to(DEV), (1, T),
                                   W)[3]
        assert np.array_equal(routes.cpu().numpy(), np.where(want_end >= 0, want_end + 1, -1))


def _latest_longest(q, k, i, W):
    """End position of the latest longest match of row i, by a look at all earlier positions."""
    j = np.flatnonzero(k[:i] == q[i])
    length = 1
    while len(j) and length < W:
        longer = j[j >= length]
        longer = longer[k[longer - length] == q[i - length]]
        if len(longer) == 0:
            break
        j, length = longer, length + 1
    return int(j[-1]) if len(j) else -1


def test_histories_beyond_the_narrow_table_entries():
    """More than 65535 steps of 16 positions: training forward, batched inference and stream."""
    import rosa_soft_b200 as rs
    from rosa_soft_b200 import cabi
    T, W, bits = 65535 * 16 + 200, 24, 8
    q, k = _streams(T, 1, bits, 9)
    q[T - 120:T - 80] = k[1000:1040]
    q[T - 60:T - 30] = k[T - 150:T - 120]
    rows = np.concatenate([np.arange(T - 300, T), np.arange(40)])
    want = np.array([_latest_longest(q[:, 0], k[:, 0], int(i), W) for i in rows])
    v = torch.randn(T, 1, 4, device=DEV)
    routes = cabi.hard_forward(_logits(q, bits), _logits(k, bits), v, (1, T), W)[3].cpu().numpy()[rows, 0]
    assert np.array_equal(routes, np.where(want >= 0, want + 1, -1))
    as_int = lambda x: torch.from_numpy(x.view(np.int32))[None].to(DEV)  # noqa: E731
    _, end = rs.rosa_hard_inference(as_int(q), as_int(k), v[None], max_suffix_length=W)
    assert np.array_equal(end[0, :, 0].cpu().numpy()[rows], want)
    byte = lambda x: torch.from_numpy(x.astype(np.uint8))[None].to(DEV)  # noqa: E731
    tq, tk = byte(q), byte(k)
    ends = []
    with rs.RosaRuntime(1, 1, bits, bits, W) as runtime:
        cuts = [0, 5000, 65535 * 16 - 8, T - 120, *range(T - 60, T, 7), T]   # prompts, then steps
        for a, b in zip(cuts[:-1], cuts[1:]):
            ends.append(runtime.update_packed(tq[:, a:b], tk[:, a:b], tk[:, a:b])[1])
    assert np.array_equal(torch.cat(ends, dim=1)[0, :, 0].cpu().numpy()[rows], want)


@pytest.mark.parametrize("bits,W,alphabet", [(1, 40, None), (1, 200, 1), (3, 2, None), (8, 32, 30), (8, 1, None)])
@pytest.mark.parametrize("form", ("packed", "float32", "bfloat16"))
def test_steps_and_chunks_of_a_stream_equal_one_pass(form, bits, W, alphabet):
    """Chunks on both sides of the 16 tokens of the one-kernel step, over two growths of the state."""
    from rosa_soft_b200 import RosaRuntime
    H, Hp, B, pay_bits = 4, 2, 2, 5
    chunks = [1, 16, 17, 15, 1, 33, 16, 16, 2, 120, 16, 1, 40, 250, 5, 16, 17]
    T = sum(chunks)
    q, k = _streams(B * T, H, bits, 3 * bits + W, alphabet)
    pay = np.random.default_rng(1).integers(0, 1 << pay_bits, size=(B * T, Hp)).astype(np.uint32)
    cu = np.arange(B + 1) * T
    want, want_end = orc.hard_inference(q, k, pay.astype(np.float32)[..., None], cu, W)
    shape = lambda x, n: x.reshape(B, T, n)  # noqa: E731
    got, ends = [], []
    runtime = RosaRuntime(H, Hp, bits, pay_bits, W)
    at = 0
    for n in chunks:
        part = [shape(x, heads)[:, at:at + n] for x, heads in ((q, H), (k, H), (pay, Hp))]
        if form == "packed":
            out, end = runtime.update_packed(*(torch.from_numpy(x.astype(np.uint8)).to(DEV) for x in part))
        else:
            dt = getattr(torch, form)
            out, end = runtime.update(_logits(part[0], bits).to(dt), _logits(part[1], bits).to(dt),
                                      _logits(part[2], pay_bits).to(dt))
            assert out.dtype == dt
        got.append(out)
        ends.append(end)
        at += n
    end = torch.cat(ends, dim=1).cpu().numpy().reshape(-1, H)
    out = torch.cat(got, dim=1).float().cpu().numpy()
    assert np.array_equal(end, want_end)
    if form == "packed":
        assert np.array_equal(out.reshape(-1, H), want[:, :, 0])
    else:
        signs = 2.0 * ((want.astype(np.int64) >> np.arange(pay_bits)) & 1) - 1.0
        signs[want_end < 0] = 0.0
        assert np.array_equal(out.reshape(-1, H, pay_bits), signs)


@pytest.mark.parametrize("dtype", (torch.float32, torch.float16, torch.bfloat16))
@pytest.mark.parametrize("packed", (False, True))
def test_native_call_equals_the_python_form(dtype, packed):
    import rosa_soft_b200 as rs
    from rosa_soft_b200 import soft
    H, D, Hv, Dv, W = 4, 5, 2, 3, 9
    lead = (70,) if packed else (2, 35)
    cu = torch.tensor([0, 20, 21, 70], dtype=torch.int32, device=DEV) if packed else None
    q, k, v, go = (nonzero_randn((*lead, *s), 40 + n, dtype).to(DEV)
                   for n, s in enumerate(((H, D), (H, D), (Hv, Dv), (H, Dv))))

    def grads(call, wanted):
        leaves = [t.clone().requires_grad_(n in wanted) for n, t in enumerate((q, k, v))]
        torch.cuda.manual_seed(11)
        out = call(*leaves)
        return [out.detach(), *torch.autograd.grad(out, [t for n, t in enumerate(leaves) if n in wanted], go)]

    controls = dict(max_suffix_length=W, scale=1.2, dropout_p=0.2, mismatch_scale=3.0)
    native = (lambda *t: rs.rosa_soft_varlen(*t, cu, **controls)) if packed else (
        lambda *t: rs.rosa_soft(*t, **controls))
    python = lambda *t: soft._run(*t, cu, min(W, lead[-1]), 1.2, 0.2, 3.0)  # noqa: E731
    for wanted in ((0, 1, 2), (0,), (2,), (1, 2)):
        for a, b in zip(grads(native, wanted), grads(python, wanted)):
            assert a.dtype == dtype and torch.equal(a, b)


def test_native_call_keeps_the_rules_of_autograd():
    import rosa_soft_b200 as rs
    q, k = (nonzero_randn((1, 24, 2, 4), s).to(DEV).requires_grad_(True) for s in (1, 2))
    v = nonzero_randn((1, 24, 2, 3), 3).to(DEV).requires_grad_(True)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t.cpu(),
                                                  lambda t: t.to(DEV)):
        out = rs.rosa_soft(q, k, v, max_suffix_length=8)
    assert len(packed) >= 5                              # q, k, v and the packed symbols
    want = torch.autograd.grad(rs.rosa_soft(q, k, v, max_suffix_length=8).sum(), (q, k, v))
    for a, b in zip(torch.autograd.grad(out.sum(), (q, k, v)), want):
        assert torch.equal(a, b)
    # once differentiable
    go = torch.ones_like(out, requires_grad=True)
    dq, = torch.autograd.grad(rs.rosa_soft(q, k, v, max_suffix_length=8), q, go, create_graph=True)
    with pytest.raises(RuntimeError, match="once_differentiable"):
        dq.sum().backward()
    # an input that was changed in place after the forward is noticed
    w = q.detach().clone().requires_grad_(True)
    leaf = w * 1.0
    out = rs.rosa_soft(leaf, k, v, max_suffix_length=8)
    leaf.add_(1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.sum().backward()


def _held(stream):
    """Queues some milliseconds of work on a stream (bounded: a spin of a fixed count of cycles)."""
    with torch.cuda.stream(stream):
        torch.cuda._sleep(20_000_000)


def _stream_case(T, seed):
    """Packed symbols [2, T, 4] (4 bits) and the result of one pass over them."""
    B, H, bits, W = 2, 4, 4, 32
    q, k = _streams(B * T, H, bits, seed)
    want, want_end = orc.hard_inference(q, k, k.astype(np.float32)[..., None], np.arange(B + 1) * T, W)
    byte = lambda x: torch.from_numpy(x.astype(np.uint8)).reshape(B, T, H).to(DEV)  # noqa: E731
    return byte(q), byte(k), want[..., 0].reshape(B, T, H), want_end.reshape(B, T, H)


def _feed(runtime, q, k, a, b, **how):
    return runtime.update_packed(q[:, a:b], k[:, a:b], k[:, a:b], **how)


def _check_stream(results, want, want_end):
    assert np.array_equal(torch.cat([r[1] for r in results], dim=1).cpu().numpy(), want_end)
    assert np.array_equal(torch.cat([r[0] for r in results], dim=1).cpu().numpy(), want)


def test_a_growth_on_another_stream_keeps_the_old_state_until_it_is_copied():
    """The growing update waits on a second stream while the first one allocates and fills blocks of
    the sizes that the old state had."""
    from rosa_soft_b200 import RosaRuntime
    T = 700
    q, k, want, want_end = _stream_case(T, 3)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    runtime = RosaRuntime(4, 4, 4, 4, 32)
    first = _feed(runtime, q, k, 0, 200)
    side = torch.cuda.Stream()
    _held(side)
    work = _feed(runtime, q, k, 200, T, stream=side, async_op=True)
    noise = [torch.full((n,), 255, dtype=torch.uint8, device=DEV)
             for n in (8, 16, 512, 2048, 8192, 16384, 65536, 131072, 262144) for _ in range(8)]
    second = work.wait()
    torch.cuda.synchronize()
    assert len(noise) == 72
    _check_stream([first, second], want, want_end)


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
@pytest.mark.parametrize("how", ("reset", "load"))
def test_a_runtime_that_was_reset_or_loaded_may_go_on_on_another_gpu(how):
    from rosa_soft_b200 import RosaRuntime
    T = 300
    q, k, want, want_end = _stream_case(T, 4)
    runtime = RosaRuntime(4, 4, 4, 4, 32)
    first = _feed(runtime, q, k, 0, 100)
    if how == "reset":
        runtime.reset()
        results = []
        at = 0
    else:
        state = {n: x.to("cuda:1") if isinstance(x, torch.Tensor) else x
                 for n, x in runtime.state_dict().items()}
        runtime.load_state_dict(state)
        results = [tuple(x.cpu() for x in first)]
        at = 100
    for a, b in ((at, 150), (150, T)):
        results.append(tuple(x.cpu() for x in _feed(runtime, q.to("cuda:1"), k.to("cuda:1"), a, b)))
    _check_stream(results, want, want_end)


def test_an_update_after_one_that_failed_in_its_growth_waits_for_the_copies():
    """The failing update grows the state on a held-back stream and then cannot allocate its result; the
    next one comes on the stream of the update before it."""
    from rosa_soft_b200 import RosaRuntime
    T = 900
    q, k, want, want_end = _stream_case(T, 5)
    runtime = RosaRuntime(4, 4, 4, 4, 32)
    first = _feed(runtime, q, k, 0, 250)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    _held(side)
    part = [x[:, 250:T].contiguous() for x in (q, k, k)]
    with torch.cuda.stream(side), pytest.raises(RuntimeError):
        runtime._core.packed(*part, [0, T - 250, 2 * (T - 250)], None, None, [-7, 4])
    assert runtime._core.capacity >= T
    second = _feed(runtime, q, k, 250, T)
    torch.cuda.synchronize()
    _check_stream([first, second], want, want_end)


def test_a_load_that_fails_leaves_a_fresh_runtime():
    from rosa_soft_b200 import RosaRuntime
    T = 120
    q, k, want, want_end = _stream_case(T, 6)
    source = RosaRuntime(4, 4, 4, 4, 32)
    source.update_packed(*(torch.cat([x, x]) for x in (q, k, k)), sequence_ids=[3, 4, 5, 6])    # four slots
    state = source.state_dict()
    runtime = RosaRuntime(4, 4, 4, 4, 32)
    for broken in ({"payload_history": state["payload_history"][..., :-1]},
                   {"key_history": state["key_history"][:2]}, {"lengths": [T] * 3}):
        with pytest.raises(RuntimeError):
            runtime.load_state_dict({**state, **broken})
        assert runtime.memory_stats()["sequences"] == 0
    _check_stream([_feed(runtime, q, k, 0, 50), _feed(runtime, q, k, 50, T)], want, want_end)    # two slots, no IDs


def test_a_state_is_saved_between_the_updates_around_it_whatever_their_streams():
    from rosa_soft_b200 import RosaRuntime
    T = 400
    q, k, want, want_end = _stream_case(T, 8)
    runtime = RosaRuntime(4, 4, 4, 4, 32)
    first = _feed(runtime, q, k, 0, 100)
    side = torch.cuda.Stream()
    _held(side)
    second = _feed(runtime, q, k, 100, 250, stream=side, async_op=True)     # no growth: capacity 256
    state = runtime.state_dict()                                            # not ordered by the caller
    loaded = RosaRuntime(4, 4, 4, 4, 32)
    loaded.load_state_dict(state)
    rest = [_feed(r, q, k, 250, T) for r in (runtime, loaded)]
    done = second.wait()
    for r in rest:
        _check_stream([first, done, r], want, want_end)


def test_host_threads_with_calls_of_different_sizes_do_not_disturb_each_other():
    """The kernels of two threads need different amounts of shared memory."""
    import threading

    import rosa_soft_b200 as rs

    def inputs(T, D, seed):
        return [nonzero_randn((1, T, 1, n), seed + s).to(DEV) for s, n in enumerate((D, D, 8))]

    # few heads are indexed in pieces: tables of 75 to 140 KB a block
    cases = [inputs(T, D, 11 * n) for n, (T, D) in enumerate([(2048, 8), (4096, 8), (8192, 8), (4096, 3)])]
    call = lambda case: rs.rosa_soft(*case, max_suffix_length=20)  # noqa: E731
    want = [call(case) for case in cases]
    torch.cuda.synchronize()
    failed = []

    def work(n):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(3000):
                    got = call(cases[n])
                torch.cuda.current_stream().synchronize()
                assert torch.equal(got, want[n])
        except Exception as error:  # noqa: BLE001
            failed.append((n, error))

    threads = [threading.Thread(target=work, args=(n,)) for n in range(len(cases))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


@pytest.mark.parametrize("bits", (1, 2))
def test_chunks_of_long_histories_of_few_heads_take_the_largest_index_blocks(bits):
    """Wide table entries, all shorter lengths, two or four pieces: 24 warps a block."""
    from rosa_soft_b200 import RosaRuntime
    held, n, W = 65535 * 16 + 40, 1100, 24
    q, k = _streams(held + n, 1, bits, 5, copies=False)
    q[held + 500:held + 560] = k[held + 100:held + 160]
    q[held + 700:held + 790] = k[3000:3090]
    byte = lambda x: torch.from_numpy(x.astype(np.uint8).reshape(1, 1, -1)).to(DEV)  # noqa: E731
    runtime = RosaRuntime(1, 1, bits, bits, W)
    config = runtime.state_dict()["config"]
    runtime.load_state_dict({"config": config, "lengths": [held], "query_history": byte(q[:held]),
                             "key_history": byte(k[:held]), "payload_history": byte(k[:held])})
    tq, tk = (byte(x[held:]).reshape(1, n, 1) for x in (q, k))
    end = runtime.update_packed(tq, tk, tk)[1][0, :, 0].cpu().numpy()
    rows = np.concatenate([np.arange(0, n, 16), np.arange(540, 560), np.arange(770, 790)])
    assert np.array_equal(end[rows], [_latest_longest(q[:, 0], k[:, 0], held + int(i), W) for i in rows])


def _few_symbols(n, heads, bits, seed, alphabet, top=None):
    """Key symbols of a small alphabet (with `top`: one symbol that often, the rest wide) and a query stream
    of other positions of the same heads."""
    rng = np.random.default_rng(seed)
    letters = rng.choice(1 << min(bits, 20), size=alphabet, replace=False).astype(np.uint32)
    k = letters[rng.integers(0, alphabet, size=(n, heads))]
    if top is not None:
        k = np.where(rng.random((n, heads)) < top, letters[0], k)
    return np.roll(k, n // 3, axis=0).astype(np.uint32), k.astype(np.uint32)


RUN_LENGTHS = (513, 40, 767, 769, 2303, 2306, 4400, 1, 600)     # around tiles of 256 rows, bands of 2048


@pytest.mark.parametrize("bits,W,alphabet,top", [
    (8, 40, 2, None), (8, 4000, 3, None), (3, 2, 2, None), (24, 128, 2, None), (16, 32, 7, None),
    (16, 32, 500, 0.9), (8, 64, 200, 0.6), (24, 600000, 2, None)])
def test_rows_on_chains_too_long_to_follow(bits, W, alphabet, top):
    """Forward over packed sequences and batched inference over the longest of them."""
    import rosa_soft_b200 as rs
    from rosa_soft_b200 import cabi
    H = 8 if bits <= 16 else 2          # tiles of 256 rows, or of 64 where those are too few
    cu = np.concatenate([[0], np.cumsum(RUN_LENGTHS)])
    parts = [_few_symbols(n, H, bits, n + W, alphabet, top) for n in RUN_LENGTHS]
    q, k = (np.concatenate([p[x] for p in parts]) for x in (0, 1))
    pay = np.random.default_rng(3).standard_normal((int(cu[-1]), 1, 4)).astype(np.float32)
    want_out, want_end = orc.hard_inference(q, k, pay, cu, W)
    device_cu = torch.from_numpy(cu.astype(np.int32)).to(DEV)
    routes = cabi.hard_forward(_logits(q, bits), _logits(k, bits), torch.from_numpy(pay).to(DEV), device_cu,
                               W)[3].cpu().numpy()
    starts = np.repeat(cu[:-1], RUN_LENGTHS)[:, None]
    assert np.array_equal(routes, np.where(want_end >= 0, want_end + 1 + starts, -1))
    s = slice(cu[6], cu[7])
    as_int = lambda x: torch.from_numpy(x[s].view(np.int32))[None].to(DEV)  # noqa: E731
    out, end = rs.rosa_hard_inference(as_int(q), as_int(k), torch.from_numpy(pay[s])[None].to(DEV),
                                      max_suffix_length=W)
    assert np.array_equal(end[0].cpu().numpy(), want_end[s]) and np.array_equal(out[0].cpu().numpy(), want_out[s])


def test_lone_rows_on_long_chains():
    """A symbol that is frequent among the keys and rare among the queries: a few pending rows a tile."""
    from rosa_soft_b200 import cabi
    T, H, bits, W = 3000, 2, 16, 32
    rng = np.random.default_rng(1)
    k = rng.integers(0, 1 << bits, size=(T, H)).astype(np.uint32)
    q = rng.integers(0, 1 << bits, size=(T, H)).astype(np.uint32)
    k[rng.random((T, H)) < 0.3] = 77
    q[::60] = 77
    q[1200:1215] = k[300:315]
    v = nonzero_randn((T, 1, 3), 5).to(DEV)
    routes = cabi.hard_forward(_logits(q, bits), _logits(k, bits), v, (1, T), W)[3]
    _, want = orc.hard_forward(_logits(q, bits).cpu().numpy(), _logits(k, bits).cpu().numpy(), v.cpu().numpy(),
                               np.array([0, T]), W)
    assert np.array_equal(routes.cpu().numpy(), np.where(want > 0, want, -1))


@pytest.mark.parametrize("bits,W,alphabet,top", [(8, 32, 2, None), (8, 300, 3, None), (2, 5, 2, None),
                                                 (8, 32, 200, 0.8)])
def test_streams_of_few_symbols_equal_one_pass(bits, W, alphabet, top):
    """Chunks around the tiles of the run matcher and single steps, slots of different lengths."""
    from rosa_soft_b200 import RosaRuntime
    H, B = 40 if bits == 2 else 3, 2
    chunks = [(700, 650), (300, 0), (1, 1), (16, 16), (17, 40), (257, 255), (2200, 2306), (40, 300), (1, 1), (7, 0)]
    T = [sum(c[s] for c in chunks) for s in range(B)]
    data = [_few_symbols(T[s], H, bits, 5 * s + W, alphabet, top) for s in range(B)]
    runtime = RosaRuntime(H, H, bits, bits, W)
    got, at = [[], []], [0, 0]
    for n in chunks:
        part = [torch.from_numpy(np.concatenate([data[s][x][at[s]:at[s] + n[s]] for s in range(B)]).astype(np.uint8))
                for x in (0, 1)]
        cu = torch.tensor([0, n[0], n[0] + n[1]], dtype=torch.int32, device=DEV)
        out, end = runtime.update_packed(part[0].to(DEV), part[1].to(DEV), part[1].to(DEV), cu)
        for s, rows in enumerate((slice(0, n[0]), slice(n[0], n[0] + n[1]))):
            got[s].append((out[rows].cpu().numpy(), end[rows].cpu().numpy()))
            at[s] += n[s]
    for s in range(B):
        q, k = data[s]
        want, want_end = orc.hard_inference(q, k, k.astype(np.float32)[..., None], np.array([0, T[s]]), W)
        assert np.array_equal(np.concatenate([g[1] for g in got[s]]), want_end)
        assert np.array_equal(np.concatenate([g[0] for g in got[s]]), want[..., 0])


@pytest.mark.parametrize("bits", (1, 8, 16))
@pytest.mark.parametrize("heads", (1, 12))        # indexed in pieces, in one
def test_packs_of_one_long_and_many_short_sequences(bits, heads):
    """Every sequence has buckets, pieces and a share of the launch by its own length: forward and gradients."""
    import rosa_soft_b200 as rs
    from tests.helpers import normalised_error, oracle_grads
    rng = np.random.default_rng(bits)
    lengths = np.concatenate([rng.integers(0, 20, size=150), [1700, 511, 512], rng.integers(1, 40, size=50)])
    cu = np.concatenate([[0], np.cumsum(lengths)])
    N, W = int(cu[-1]), 24
    q, k = _streams(N, heads, bits, 7)
    leaves = [t.requires_grad_(True) for t in (_logits(q, bits), _logits(k, bits),
                                               nonzero_randn((N, 1, 4), 5).to(DEV))]
    out = rs.rosa_soft_varlen(*leaves, torch.from_numpy(cu.astype(np.int32)).to(DEV), max_suffix_length=W,
                              dropout_p=0.0)
    go = nonzero_randn((N, heads, 4), 6).to(DEV)
    got = torch.autograd.grad(out, leaves, go)
    host = [t.detach().cpu().numpy() for t in leaves]
    assert np.array_equal(out.detach().cpu().numpy(), orc.hard_forward(*host, cu, W)[0])
    want = oracle_grads(*leaves, go, cu, W, 1.0, 0.0, 3.0, 0)
    for mine, ref in zip(got, want):
        assert normalised_error(mine.cpu().numpy(), ref) <= 1e-4       # the bound of float32 inputs
