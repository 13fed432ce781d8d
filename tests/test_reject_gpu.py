"""Rejection-sampling acceptance over a draft tree: the CUDA kernel against the
CPU oracle's statement of the same rule, through the C ABI.

The reference verifies greedily only (engine/speculative.go:73-75), so nothing in
it pins this rule; the pins are the oracle (integer-exact rule, bit-exact match
demanded here) and two properties: a temperature near zero with one-hot draft
distributions reproduces the greedy walk, and the committed position advances
by accepted + 1.
"""
import numpy as np
import pytest

from oracle import pyoracle as yo
from yuuka_b200 import cuda, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tiny():
    cfg = synth.tiny_config()
    tensors = synth.make_model(cfg, "q8_0", seed=7, unit_norms=False)
    dev = cuda.Device(0)
    gm = cuda.Model(dev, cfg, tensors)
    yield cfg, gm, dev
    gm.close()
    dev.close()


def softmax32(x):
    x = x.astype(np.float64)
    e = np.exp(x - x.max(axis=-1, keepdims=True))
    return (e / e.sum(axis=-1, keepdims=True)).astype(np.float32)


def draft_tree(rng, logits, parent, temperature, noise):
    """Draft distributions q[c] = softmax((L[parent c] + noise) / T) and tokens drawn from them."""
    n, V = logits.shape
    q = np.zeros((n, V), np.float32)
    tokens = np.zeros(n, np.int32)
    for c in range(1, n):
        q[c] = softmax32((logits[parent[c]] + noise * rng.standard_normal(V).astype(np.float32)) / temperature)
        tokens[c] = rng.choice(V, p=q[c].astype(np.float64) / q[c].astype(np.float64).sum())
    return q, tokens


@pytest.mark.parametrize("temperature,noise", [(0.8, 1.0), (0.7, 0.0), (1.5, 3.0)])
def test_rejection_walk_matches_oracle_bit_for_bit(tiny, temperature, noise):
    cfg, gm, dev = tiny
    V, B = cfg["vocab"], 3
    parent = np.array(synth.tree_16(), np.int32)
    N = parent.size
    rng = np.random.default_rng(int(temperature * 100) + int(noise * 10))
    sess = cuda.Session(gm, max_batch=B, max_nodes=N, capacity=128, kv_format=cuda.KV_F16)
    prompts = [synth.uniform_i32(20 + 7 * b, 0, V, 60 + b) for b in range(B)]
    pend = [int(np.argmax(sess.forward(prompts[b], seq=b))) for b in range(B)]
    # a first pass that commits nothing gives the logits of the root rows; drafts are drawn level by level
    tokens = np.zeros((B, N), np.int32)
    tokens[:, 0] = pend
    q = np.zeros((B, N, V), np.float32)
    depth = np.zeros(N, np.int32)
    for c in range(1, N):
        depth[c] = depth[parent[c]] + 1
    for level in range(1, int(depth.max()) + 1):
        res = sess.verify(tokens, parent=parent, mode=cuda.ACCEPT_NONE, want_logits=True)
        for b in range(B):
            for c in np.nonzero(depth == level)[0]:
                q[b, c] = softmax32((res.logits[b, parent[c]] + noise * rng.standard_normal(V).astype(np.float32)) / temperature)
                p64 = q[b, c].astype(np.float64)
                tokens[b, c] = rng.choice(V, p=p64 / p64.sum())
    logits = sess.verify(tokens, parent=parent, mode=cuda.ACCEPT_NONE, want_logits=True).logits
    uniforms = rng.random((B, N, 2), dtype=np.float32)
    uniforms = np.minimum(uniforms, np.float32(0.99999994))
    qbuf = dev.upload(q)
    pos_before = [sess.position(b) for b in range(B)]
    res = sess.verify(tokens, parent=parent, mode=cuda.ACCEPT_REJECTION, temperature=temperature, draft_probs=qbuf,
                      uniforms=uniforms, want_logits=True)
    assert np.array_equal(res.logits.view(np.uint32), logits.view(np.uint32))  # the step is deterministic
    total_accepted = 0
    for b in range(B):
        a, path, emitted = yo.accept_rejection_tree(logits[b], q[b], tokens[b], parent, temperature, uniforms[b])
        assert int(res.accepted[b]) == a
        assert res.path[b, :a].tolist() == path.tolist()
        assert res.emitted[b, :a + 1].tolist() == emitted.tolist()
        assert sess.position(b) == pos_before[b] + a + 1
        total_accepted += a
    if noise <= 1.0:
        assert total_accepted > 0  # the case exercises the accept branch, not only the residual draw
    qbuf.free()
    sess.close()


def test_cold_temperature_with_one_hot_drafts_is_the_greedy_walk(tiny):
    cfg, gm, dev = tiny
    V = cfg["vocab"]
    parent = np.array(synth.tree_16(), np.int32)
    N = parent.size
    prompt = synth.uniform_i32(33, 0, V, 91)
    outs = []
    for mode in (cuda.ACCEPT_GREEDY, cuda.ACCEPT_REJECTION):
        sess = cuda.Session(gm, max_batch=1, max_nodes=N, capacity=128, kv_format=cuda.KV_F32)
        pend = int(np.argmax(sess.forward(prompt)))
        tokens = synth.uniform_i32(N, 0, V, 92)
        tokens[0] = pend
        # make a three-deep greedy path exist in the tree: rows 2, 8, 12
        for row in (2, 8, 12):
            lg = sess.verify([tokens], parent=parent, mode=cuda.ACCEPT_NONE, want_logits=True).logits[0]
            tokens[row] = int(np.argmax(lg[parent[row]]))
        if mode == cuda.ACCEPT_GREEDY:
            res = sess.verify([tokens], parent=parent)
        else:
            q = np.zeros((1, N, V), np.float32)
            q[0, np.arange(N), tokens] = 1.0
            qbuf = dev.upload(q)
            u = np.full((1, N, 2), 0.5, np.float32)
            res = sess.verify([tokens], parent=parent, mode=mode, temperature=0.01, draft_probs=qbuf, uniforms=u)
            qbuf.free()
        a = int(res.accepted[0])
        outs.append((a, res.path[0, :a].tolist(), res.emitted[0, :a + 1].tolist(), sess.position()))
        sess.close()
    assert outs[0] == outs[1]
    assert outs[0][0] == 3 and outs[0][1] == [2, 8, 12]


def test_rejection_arguments_are_validated(tiny):
    cfg, gm, dev = tiny
    V = cfg["vocab"]
    sess = cuda.Session(gm, max_batch=1, max_nodes=4, capacity=64, kv_format=cuda.KV_F32)
    sess.forward([1, 2, 3], want_logits=False)
    toks = [[5, 6, 7, 8]]
    q = dev.upload(np.zeros((1, 4, V), np.float32))
    small = dev.upload(np.zeros(16, np.float32))
    u = np.full((1, 4, 2), 0.5, np.float32)
    bad = [dict(temperature=0.0, draft_probs=q, uniforms=u), dict(temperature=0.8, draft_probs=None, uniforms=u),
           dict(temperature=0.8, draft_probs=small, uniforms=u), dict(temperature=0.8, draft_probs=q, uniforms=None),
           dict(temperature=0.8, draft_probs=q, uniforms=np.full((1, 4, 2), 1.0, np.float32))]
    for kw in bad:
        with pytest.raises(cuda.YuukaError) as e:
            sess.verify(toks, mode=cuda.ACCEPT_REJECTION, **kw)
        assert e.value.status == 1
    assert sess.position() == 3  # nothing ran
    q.free(); small.free()
    sess.close()


def test_acceptance_case_of_the_kernel_microbenchmark_matches_the_oracle():
    """fp32 logits N(0, 3) over 248,320 tokens for 16 sequences x 9 positions (the microbenchmark names 64
    sequences; 16 keep the CPU side of the test to seconds), draft probabilities = softmax of the logits plus
    N(0, 1) noise, temperature 0.7, seeded uniforms: yuuka_accept_tree returns the oracle's accepted counts,
    paths and emitted tokens bit for bit, for the rejection walk and for the greedy walk."""
    V, B, N, T = 248320, 16, 9, 0.7
    dev = cuda.Device(0)
    stream = dev.stream()
    rng = np.random.default_rng(2026)
    logits = (3.0 * rng.standard_normal((B, N, V), dtype=np.float32)).astype(np.float32)
    parent = np.arange(-1, N - 1, dtype=np.int32)
    q = np.zeros((B, N, V), np.float32)
    tokens = np.zeros((B, N), np.int32)
    tokens[:, 0] = rng.integers(0, V, B)
    for b in range(B):
        for c in range(1, N):
            q[b, c] = softmax32(logits[b, c - 1] / T + rng.standard_normal(V, dtype=np.float32))
            # half of the drafts are the draft model's most likely token, half are drawn from it
            if (b + c) % 2:
                tokens[b, c] = int(np.argmax(q[b, c]))
            else:
                p64 = q[b, c].astype(np.float64)
                tokens[b, c] = rng.choice(V, p=p64 / p64.sum())
    uniforms = np.minimum(rng.random((B, N, 2), dtype=np.float32), np.float32(0.99999994))
    lb, qb = dev.upload(logits), dev.upload(q)
    acc, em, path = cuda.accept_tree(stream, lb, tokens, V, parent=parent, mode=cuda.ACCEPT_REJECTION, temperature=T,
                                     draft_probs=qb, uniforms=uniforms)
    total = 0
    for b in range(B):
        a, p_o, e_o = yo.accept_rejection_tree(logits[b], q[b], tokens[b], parent, T, uniforms[b])
        assert int(acc[b]) == a, b
        assert path[b, :a].tolist() == p_o.tolist() and em[b, :a + 1].tolist() == e_o.tolist()
        total += a
    assert 0 < total < B * (N - 1)
    # greedy walk over the same logits, with the first three drafts of every other sequence set to the argmax chain
    for b in range(0, B, 2):
        for c in range(1, 4):
            tokens[b, c] = int(np.argmax(logits[b, c - 1]))
    acc, em, path = cuda.accept_tree(stream, lb, tokens, V, parent=parent)
    for b in range(B):
        a, p_o, e_o = yo.accept_greedy_tree(logits[b], tokens[b], parent)
        assert int(acc[b]) == a and path[b, :a].tolist() == p_o.tolist() and em[b, :a + 1].tolist() == e_o.tolist()
        assert a >= 3 or b % 2
    lb.free(); qb.free()
    stream.destroy()
    dev.close()


@pytest.mark.parametrize("B,V", [(2, 1000), (2, 4099), (2, 8192), (3, 32767), (2, 32768), (40, 65536), (80, 65538), (2, 262147)])
def test_rejection_walk_at_the_vocabulary_sizes_where_the_launch_changes(B, V):
    """One CTA, two, four and eight CTAs per sequence, vocabularies that 16-byte loads do not divide: trees of 17
    rows, bit for bit the oracle's."""
    parent, T = synth.tree_16(), 0.8
    N = parent.size
    dev = cuda.Device(0)
    stream = dev.stream()
    rng = np.random.default_rng(V)
    logits = (3.0 * rng.standard_normal((B, N, V), dtype=np.float32)).astype(np.float32)
    q, tokens = np.zeros((B, N, V), np.float32), np.zeros((B, N), np.int32)
    for b in range(B):
        if b >= 3:  # (many sequences: copies of the first three)
            logits[b], q[b], tokens[b] = logits[b % 3], q[b % 3], tokens[b % 3]
            continue
        for c in range(1, N):
            q[b, c] = softmax32((logits[b, parent[c]] + rng.standard_normal(V, dtype=np.float32)) / T)
            tokens[b, c] = int(np.argmax(q[b, c])) if (b + c) % 2 else rng.integers(0, V)
    uniforms = np.minimum(rng.random((B, N, 2), dtype=np.float32), np.float32(0.99999994))
    lb, qb = dev.upload(logits), dev.upload(q)
    for _ in range(2):  # the second call reuses what the first left in the stream's scratch
        acc, em, path = cuda.accept_tree(stream, lb, tokens, V, parent=np.tile(parent, (B, 1)), mode=cuda.ACCEPT_REJECTION,
                                         temperature=T, draft_probs=qb, uniforms=uniforms)
        for b in (range(B) if B < 4 else (0, 1, 2, B - 1)):
            a, p_o, e_o = yo.accept_rejection_tree(logits[b], q[b], tokens[b], parent, T, uniforms[b])
            assert int(acc[b]) == a, b
            assert path[b, :a].tolist() == p_o.tolist() and em[b, :a + 1].tolist() == e_o.tolist()
            assert (path[b, a:] == -1).all() and (em[b, a + 1:] == -1).all()
    lb.free(); qb.free()
    stream.destroy()
    dev.close()


@pytest.mark.parametrize("V", [1000, 4099, 65536, 262147])
@pytest.mark.parametrize("T", [0.8, 1e-39])   # 1 / 1e-39 overflows: only the maximum keeps weight
def test_infinite_logits_take_all_the_weight(V, T):
    """A chain whose first row has +infinity at the drafted token (accepted) and whose second has it at another one
    (the draft is rejected, that token emitted); masked tokens at -infinity and at the lowest float."""
    N, B = 4, 2
    rng = np.random.default_rng(V)
    logits = rng.standard_normal((B, N, V), dtype=np.float32)
    logits[:, :, rng.choice(V, V // 3, replace=False)] = -np.inf
    logits[1][:, rng.choice(V, V // 3, replace=False)] = np.finfo(np.float32).min
    q = np.zeros((B, N, V), np.float32)
    tokens = np.zeros((B, N), np.int32)
    for b in range(B):
        hot = rng.choice(V, 2, replace=False)
        logits[b, 0, hot[0]] = logits[b, 1, hot[1]] = np.inf
        tokens[b, 1:] = hot[0]
        q[b, :, hot[0]] = 0.9
    uniforms = np.full((B, N, 2), 0.5, np.float32)
    parent = np.arange(-1, N - 1, dtype=np.int32)
    dev = cuda.Device(0)
    stream = dev.stream()
    lb, qb = dev.upload(logits), dev.upload(q)
    acc, em, path = cuda.accept_tree(stream, lb, tokens, V, mode=cuda.ACCEPT_REJECTION, temperature=T, draft_probs=qb,
                                     uniforms=uniforms)
    for b in range(B):
        a, p_o, e_o = yo.accept_rejection_tree(logits[b], q[b], tokens[b], parent, T, uniforms[b])
        assert a == 1 and e_o.tolist() == [int(tokens[b, 1]), int(np.argmax(logits[b, 1]))]
        assert int(acc[b]) == a and path[b, :a].tolist() == p_o.tolist() and em[b, :a + 1].tolist() == e_o.tolist()
    lb.free(); qb.free()
    stream.destroy()
    dev.close()


@pytest.mark.parametrize("B,N,V", [(1, 64, 4099), (2, 20, 65538), (3, 33, 32768), (9, 18, 248320)])
def test_nodes_with_many_children(B, N, V):
    """Most drafts are children of the root, the others of its last child; the walk stores its weights from a second
    rejection on. Some draft rows take everything away, after which the target's own weights count again (sequence 0);
    in the others the best token keeps its weight, so that the last child is reached and accepted."""
    T = 0.9
    rng = np.random.default_rng(N)
    parent = np.zeros(N, np.int32)
    parent[0], parent[N - 6:] = -1, N - 7
    seqs = min(B, 3)
    logits = (3.0 * rng.standard_normal((seqs, N, V), dtype=np.float32)).astype(np.float32)
    q, tokens = np.zeros((seqs, N, V), np.float32), np.zeros((seqs, N), np.int32)
    for b in range(seqs):
        p = softmax32(logits[b, :1] / T)[0], softmax32(logits[b, N - 7:N - 6] / T)[0]
        for c in range(1, N):
            q[b, c] = p[c >= N - 6] * np.float32(2.0 if (b + c) % 11 == 5 else rng.uniform(0.02, 0.3))
            tokens[b, c] = rng.integers(0, V)
            if c != N - 7: q[b, c, tokens[b, c]] = 0.5  # (much against the target's weight: rejected)
        tokens[b, N - 7] = best = int(np.argmax(logits[b, 0]))
        q[b, N - 7, best] = 1e-6
        if b: q[b, 1:N - 7, best] = 0.0
    uniforms = np.minimum(rng.random((B, N, 2), dtype=np.float32) * 0.1 + 0.89, np.float32(0.99999994))
    tile = [b % seqs for b in range(B)]
    dev = cuda.Device(0)
    stream = dev.stream()
    lb, qb = dev.upload(logits[tile]), dev.upload(q[tile])
    acc, em, path = cuda.accept_tree(stream, lb, tokens[tile], V, parent=np.tile(parent, (B, 1)), mode=cuda.ACCEPT_REJECTION,
                                     temperature=T, draft_probs=qb, uniforms=uniforms)
    deep = 0
    for b in range(B):
        a, p_o, e_o = yo.accept_rejection_tree(logits[tile[b]], q[tile[b]], tokens[tile[b]], parent, T, uniforms[b])
        assert int(acc[b]) == a and path[b, :a].tolist() == p_o.tolist() and em[b, :a + 1].tolist() == e_o.tolist(), b
        deep += a > 0
    assert deep > 0 or B == 1
    lb.free(); qb.free()
    stream.destroy()
    dev.close()


def test_session_step_with_many_children(tiny):
    cfg, gm, dev = tiny
    V, N, B = cfg["vocab"], 18, 2
    rng = np.random.default_rng(8)
    parent = np.zeros(N, np.int32)
    parent[0] = -1
    sess = cuda.Session(gm, max_batch=B, max_nodes=N, capacity=64, kv_format=cuda.KV_F32)
    tokens = rng.integers(0, V, (B, N)).astype(np.int32)
    logits = sess.verify(tokens, parent=parent, mode=cuda.ACCEPT_NONE, want_logits=True).logits
    q = np.repeat(softmax32(logits[:, :1] / 0.8) * np.float32(0.2), N, 1)
    np.put_along_axis(q, tokens[:, :, None].astype(np.int64), np.float32(0.6), 2)
    uniforms = np.full((B, N, 2), 0.97, np.float32)
    qbuf = dev.upload(q)
    res = sess.verify(tokens, parent=parent, mode=cuda.ACCEPT_REJECTION, temperature=0.8, draft_probs=qbuf, uniforms=uniforms)
    for b in range(B):
        a, p_o, e_o = yo.accept_rejection_tree(logits[b], q[b], tokens[b], parent, 0.8, uniforms[b])
        assert int(res.accepted[b]) == a and res.path[b, :a].tolist() == p_o.tolist()
        assert res.emitted[b, :a + 1].tolist() == e_o.tolist()
    qbuf.free()
    sess.close()
