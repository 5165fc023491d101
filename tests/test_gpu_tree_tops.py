"""The launches that end a tree and the FRI phase (a CTA or a cluster, four lanes per hash): every
stored node at the sizes where the launches and cluster sizes change, and whole proofs whose FRI tail
starts at each layer size, with one and with eight CTAs; the proof-of-work rounds of easy targets."""
import struct

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
P = 2**31 - 1


@pytest.mark.parametrize("log", [8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18, 19])
def test_every_layer(ctx, log):
    import torch
    cols = np.random.default_rng(log).integers(0, P, size=(3, 1 << log), dtype=np.uint32)
    layers = torch.empty(((2 << log) - 1) * 32, dtype=torch.uint8, device="cuda")
    root = ctx.merkle_commit(torch.from_numpy(cols.view(np.int32)).cuda(), log, 3, layers)
    ref = np.concatenate(oracle.merkle_layers(list(cols)))
    assert np.array_equal(layers.cpu().numpy().reshape(-1, 32), ref) and root == ref[-1].tobytes()


@pytest.mark.parametrize("log_n,last", [(4, 0), (7, 0), (8, 0), (9, 2), (12, 0), (13, 1), (14, 0)])
def test_fri_tail(ctx, log_n, last):
    import stwo_b200 as sb
    o = oracle.config("functional", log_last_layer_degree_bound=last)
    g = sb.PcsConfig(o.pow_bits, sb.FriConfig(o.log_blowup_factor, last, o.n_queries))
    got = ctx.prove_wide_fibonacci(sb.Statement(log_n, 5), g, trace_kind=sb.TRACE_SEEDED, trace_seed=log_n)
    assert got == oracle.prove_wide_fib(log_n, 5, o, trace_kind=1, trace_seed=log_n)


def test_roots_read_by_more_threads_than_slots(ctx):
    """Roots come back through page-locked slots, and directly where every slot is taken: 48 threads on streams of
    their own, each with its own columns."""
    import threading
    import torch
    logs = [6 + i % 7 for i in range(48)]
    cols = [np.random.default_rng(i).integers(0, P, size=(2, 1 << log), dtype=np.uint32) for i, log in enumerate(logs)]
    want = [oracle.merkle_root(list(c)) for c in cols]
    dev = [torch.from_numpy(c.view(np.int32)).cuda() for c in cols]
    torch.cuda.synchronize()
    wrong, start = [], threading.Barrier(48)

    def work(i):
        stream = torch.cuda.Stream()
        layers = torch.empty(((2 << logs[i]) - 1) * 32, dtype=torch.uint8, device="cuda")
        start.wait()
        for _ in range(50):
            if ctx.merkle_commit(dev[i], logs[i], 2, layers, stream=stream) != want[i]:
                wrong.append(i)
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(48)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_fri_tails_of_many_proofs_in_flight(ctx):
    """Eight proofs' tails and tree tops beside other proofs' grinds: a cluster's CTAs start apart from one another,
    and each has to read the channel's state before the first one moves it on."""
    import stwo_b200 as sb
    o = oracle.config("functional", pow_bits=22)
    g = sb.PcsConfig(o.pow_bits, sb.FriConfig(o.log_blowup_factor, o.log_last_layer_degree_bound, o.n_queries))
    requests = [{"statement": sb.Statement(12 + i % 3, 5), "config": g, "trace_kind": sb.TRACE_SEEDED, "trace_seed": 90 + i}
                for i in range(24)]
    want = [oracle.prove_wide_fib(12 + i % 3, 5, o, trace_kind=1, trace_seed=90 + i) for i in range(24)]
    for _ in range(4):
        assert ctx.prove_wide_fibonacci_batch(requests, max_in_flight=8) == want


@pytest.mark.parametrize("bits", [3, 11, 16, 18, 20, 21, 22])
def test_grind_round_shapes(ctx, bits):
    """Targets whose rounds have one nonce a thread, several, a full round's grid; the lowest nonce each time."""
    for i in range(3):
        digest = bytes((i * 53 + bits + k) & 0xFF for k in range(32))
        prefix = oracle.blake2s(struct.pack("<I", 0x12345678) + b"\0" * 12 + digest + struct.pack("<I", bits))
        assert ctx.pow_grind(prefix, bits) == oracle.pow_grind(digest, bits, 8)
