"""Decode steps through the resident kernel (csrc/decode_layers.cu): against the plain oracle where its tiles, pages, pairs and
rows end, against the part-by-part path for what the oracle has no word for, and which steps it leaves alone."""
import numpy as np
import pytest
import torch

from helpers import assert_close, load_plain, make_model_dir, plain_logits, rand_tokens

pytestmark = pytest.mark.gpu

BASE = {
    "architectures": ["LlamaForCausalLM"], "model_type": "llama", "num_hidden_layers": 4, "hidden_size": 512,
    "intermediate_size": 1024, "num_attention_heads": 8, "num_key_value_heads": 2, "head_dim": 64, "vocab_size": 600,
    "rms_norm_eps": 1e-5, "rope_theta": 10000.0, "max_position_embeddings": 4096, "tie_word_embeddings": False,
    "attention_bias": False, "mlp_bias": False, "hidden_act": "silu",
}
MODELS = {
    "heads of 64": BASE,
    # one kv head for eight heads, k that ends inside a chunk of 1,024, shares of one and of two tiles
    "heads of 128, one kv head": dict(BASE, hidden_size=1152, intermediate_size=1408, num_key_value_heads=1, head_dim=128,
                                      vocab_size=2400, tie_word_embeddings=True),
    "a kv head per head": dict(BASE, hidden_size=1024, intermediate_size=2688, num_key_value_heads=8, head_dim=128),
}
# lengths in front of the decoded tokens: page and block edges, pairs that are cut over blocks, one to sixteen rows
BATCHES = [(30,), (1,), (64, 63, 65), (16, 17, 128, 15, 1, 2, 127, 300), (700, 5), (1300,),
           (9, 64, 200, 31, 32, 33, 70, 129, 4), tuple(range(3, 51, 3))]


@pytest.fixture(autouse=True)
def launches(monkeypatch):
    """These tests are of the kernel: it takes every step it can run, not only those that are shorter in it.  The rows of its
    launches, in their order (a step that is captured is launched twice: once to warm up)."""
    from stratum_b200 import kernels as K
    from stratum_b200.engine import resident
    monkeypatch.setattr(resident, "pays", lambda *a: True)
    seen, real = [], K.decode_layers

    def counted(x, *args):
        seen.append(x.shape[0])
        return real(x, *args)

    monkeypatch.setattr(K, "decode_layers", counted)
    return seen


@pytest.fixture(scope="module", params=sorted(MODELS))
def model(request, tmp_path_factory):
    path = make_model_dir(str(tmp_path_factory.mktemp("resident")), MODELS[request.param], seed=3, dtype="bfloat16")
    cfg, w = load_plain(path)
    return path, cfg, w


def _stratum(path, max_tokens):
    from stratum_b200 import Stratum
    return Stratum(path, dtype="bfloat16", max_tokens=max_tokens, max_seqs=20)


def _fill(llm, prompts):
    from stratum_b200 import StepEntry
    slots = [llm.acquire() for _ in prompts]
    for s, p in zip(slots, prompts):
        llm.engine.step([StepEntry(s, p, [])])
    return slots


def _decode(llm, slots, tokens):
    return llm.decode_step(slots, tokens, with_logits=True)[2].cpu().numpy()


@pytest.mark.parametrize("lens", BATCHES, ids=lambda b: f"{len(b)} rows, {max(b)}")
def test_against_the_oracle(model, lens, launches):
    path, cfg, w = model
    llm = _stratum(path, sum(n + 128 for n in lens))
    rng = np.random.default_rng(len(lens))
    steps = 3
    toks = [rand_tokens(rng, n + steps, cfg["vocab_size"]) for n in lens]
    slots = _fill(llm, [t[:n] for t, n in zip(toks, lens)])
    del launches[:]                                          # (a prompt of one token is a step of its own)
    got = [_decode(llm, slots, [t[n + i] for t, n in zip(toks, lens)]) for i in range(steps)]
    assert llm.model.resident_steps() is not None
    rows = len(lens) if len(lens) <= 8 else 16
    assert launches and set(launches) == {rows}
    for j, (t, n) in enumerate(zip(toks, lens)):
        ref = plain_logits(cfg, w, t)
        assert_close(np.stack([g[j] for g in got]), ref[n:], "bfloat16", f"row {j} of {n} tokens")


def test_window_and_rows_alone(model, launches):
    """A sliding window (the same attribute both paths read) against the part-by-part path, and a row's bits in another batch."""
    path, cfg, _ = model
    lens = [200, 64, 10, 130]
    rng = np.random.default_rng(1)
    toks = [rand_tokens(rng, n + 1, cfg["vocab_size"]) for n in lens]
    out = []
    for on in (True, False):
        llm = _stratum(path, 2048)
        if not on:                                           # (this model runs part by part)
            llm.model._resident, llm.model._resident_asked = None, True
        slots = _fill(llm, [t[:-1] for t in toks])
        for layer in llm.model.layers:
            layer.part("mixer").window = 70
        out.append(_decode(llm, slots, [t[-1] for t in toks]))
        assert (llm.model.resident_steps() is not None) == on
        assert launches == [4, 4]                            # (none by the second model)
    assert_close(out[0], out[1], "bfloat16", "window")
    llm = _stratum(path, 2048)
    alone = []
    for t in toks:
        slots = _fill(llm, [t[:-1]])
        alone.append(_decode(llm, slots, [t[-1]])[0])
        llm.release(slots[0])
    slots = _fill(llm, [t[:-1] for t in toks])
    both = _decode(llm, slots, [t[-1] for t in toks])
    # (pairs of up to eight pages are never cut, so the order of every sum is the same)
    assert np.array_equal(both, np.stack(alone))
    # and among twelve rows, of which the kernel takes sixteen with a second accumulator
    more = _fill(llm, [rand_tokens(rng, n, cfg["vocab_size"]) for n in (1, 63, 90, 17, 40, 128, 33, 7)])
    for s in slots:
        llm.release(s)
    slots = _fill(llm, [t[:-1] for t in toks])
    order = more[:5] + slots + more[5:]
    twelve = _decode(llm, order, [9] * 5 + [t[-1] for t in toks] + [9] * 3)
    assert launches[-1] == 16 and np.array_equal(twelve[5:9], np.stack(alone))


def test_steps_it_leaves_alone(model, launches):
    """Some rows' logits only; more rows than sixteen run part by part; a step launched from the host gives a replayed one's
    bits."""
    from stratum_b200 import StepEntry
    path, cfg, w = model
    llm = _stratum(path, 4096)
    rng = np.random.default_rng(2)
    toks = [rand_tokens(rng, 22, cfg["vocab_size"]) for _ in range(17)]
    ref = [plain_logits(cfg, w, t) for t in toks[:3]]
    slots = _fill(llm, [t[:19] for t in toks])
    got = llm.engine.step([StepEntry(s, [t[19]], [0] if i != 1 else []) for i, (s, t) in enumerate(zip(slots, toks[:3]))])
    assert_close(got.cpu().numpy(), np.stack([ref[0][19], ref[2][19]]), "bfloat16", "wanted rows")
    assert launches == [3]
    _decode(llm, slots[3:], [t[19] for t in toks[3:]])
    assert set(launches[1:]) == {16}
    del launches[:]
    got = _decode(llm, slots, [t[20] for t in toks])
    assert not launches
    assert_close(got[:3], np.stack([r[20] for r in ref]), "bfloat16", "seventeen rows")
    for s in slots:
        llm.release(s)
    a, b = _fill(llm, [t[:19] for t in toks[:2]]), _fill(llm, [t[:19] for t in toks[:2]])
    replayed = _decode(llm, a, [t[19] for t in toks[:2]])
    launched = llm.engine.step([StepEntry(s, [t[19]], [0]) for s, t in zip(b, toks)]).cpu().numpy()
    assert np.array_equal(replayed, launched) and launches == [2, 2, 2]


def test_the_cache_does_not_follow_from_the_wanted_rows(model):
    """Whose logits a caller asks for changes neither a step's keys and values nor the logits it gives."""
    from stratum_b200 import StepEntry
    path, cfg, _ = model
    llm = _stratum(path, 4096)
    rng = np.random.default_rng(4)
    toks = [rand_tokens(rng, n + 2, cfg["vocab_size"]) for n in (70, 19, 130)]
    group = llm.engine.cache.groups[0]
    left = []
    for wants in ([[0], [0], [0]], [[], [0], []], [[], [], []]):
        slots = _fill(llm, [t[:-2] for t in toks])
        got = llm.engine.step([StepEntry(s, [t[-2]], w) for s, t, w in zip(slots, toks, wants)])
        assert got.shape == (sum(map(len, wants)), cfg["vocab_size"])
        pages = [llm.engine.cache.page_table_rows([s], 0)[0] for s in slots]
        kv = [(group.k[:, p, :, (len(t) - 2) % 64].cpu(), group.v[:, p, :, (len(t) - 2) % 64].cpu())
              for p, t in zip([row[-1] for row in pages], toks)]
        nxt = _decode(llm, slots, [t[-1] for t in toks])
        left.append((got.cpu(), kv, nxt))
        for s in slots:
            llm.release(s)
    full = left[0][0]
    assert torch.equal(left[1][0], full[1:2])
    for _, kv, nxt in left[1:]:
        for (k0, v0), (k1, v1) in zip(left[0][1], kv):
            assert torch.equal(k0, k1) and torch.equal(v0, v1)
        assert np.array_equal(left[0][2], nxt)


def test_a_model_goes_with_its_last_reference(model):
    """The plan holds nothing that holds the model: no collector is needed to give its weights back."""
    import gc
    import weakref
    path, cfg, _ = model
    llm = _stratum(path, 256)
    _decode(llm, _fill(llm, [[1, 2, 3]]), [4])
    assert llm.model.resident_steps() is not None
    ref = weakref.ref(llm.model)
    gc.disable()
    try:
        del llm
        assert ref() is None
    finally:
        gc.enable()


def test_a_launch_that_is_refused(model, monkeypatch):
    """Where the blocks cannot all be resident the step runs part by part, launched and replayed, with the same bits as a model
    that never took the kernel."""
    from stratum_b200 import StepEntry
    from stratum_b200 import kernels as K
    path, cfg, _ = model
    rng = np.random.default_rng(6)
    toks = [rand_tokens(rng, n + 2, cfg["vocab_size"]) for n in (33, 5)]
    asked, real, out = [], K._fn, []
    for refused in (True, False):
        llm = _stratum(path, 1024)
        if refused:
            monkeypatch.setattr(K, "_fn", lambda lib, name, types: (lambda *a: asked.append(name) or -6)
                                if name == "stratum_decode_layers" else real(lib, name, types))
        else:
            monkeypatch.setattr(K, "_fn", real)
            llm.model._resident, llm.model._resident_asked = None, True
        slots = _fill(llm, [t[:-2] for t in toks])
        first = llm.engine.step([StepEntry(s, [t[-2]], [0]) for s, t in zip(slots, toks)]).cpu().numpy()
        out.append((first, _decode(llm, slots, [t[-1] for t in toks])))
    assert asked == ["stratum_decode_layers"]             # asked once, and not inside a capture
    for a, b in zip(*out):
        assert np.array_equal(a, b)


# The widths the kernel serves, four layers of them.  On 148 SMs: two tiles of the stream a block (widths above 2,368), three and
# four chunks of k, 5 to 9 tiles of the head (several groups of the partial sums' tiles), a k of the down product that ends
# inside a chunk, 3, 4 and 1 query heads a kv head.
WIDE = {
    "8B": dict(BASE, hidden_size=4096, intermediate_size=14336, num_attention_heads=32, num_key_value_heads=8, head_dim=128,
               vocab_size=10000, max_position_embeddings=16384),
    "7B": dict(BASE, hidden_size=4096, intermediate_size=11008, num_attention_heads=32, num_key_value_heads=32, head_dim=128,
               vocab_size=3000, max_position_embeddings=16384),
    "3B": dict(BASE, hidden_size=3072, intermediate_size=8192, num_attention_heads=24, num_key_value_heads=8, head_dim=128,
               vocab_size=12800, max_position_embeddings=16384),
    "1B": dict(BASE, hidden_size=2048, intermediate_size=8192, num_attention_heads=32, num_key_value_heads=8, head_dim=64,
               vocab_size=20000, max_position_embeddings=16384),
}
# rows; lengths.  The long ones: a block's share of 3 to 60 pages, cuts at odd pages, blocks that end one cut pair, take whole
# ones and begin another, pairs of eight and nine pages beside each other
WIDE_BATCHES = [(201,), (3700,) * 8, (64, 63, 65, 1, 512, 513, 577, 130, 30), tuple(range(20, 500, 30)),
                (9000,), (3705, 1000, 64, 2050, 513), (520, 8000, 449, 2, 575, 1090, 300, 5)]


@pytest.fixture(scope="module", params=sorted(WIDE))
def wide(request):
    from stratum_b200 import Stratum
    from stratum_b200.config import LlamaConfig
    llm = Stratum.from_random(LlamaConfig.from_dict(WIDE[request.param]), seed=5, max_tokens=64000, max_seqs=40)
    for layer in llm.model.layers:         # the attention's share of the stream, the mean of many values, is not to drown beside
        layer.part("feed_forward").down.weight.mul_(0.1)       # the feed-forward's: a page left out would not be seen then
    return llm


@pytest.mark.parametrize("lens", WIDE_BATCHES, ids=lambda b: f"{len(b)} rows, {max(b)}")
def test_served_widths(wide, lens, launches):
    """Logits of two steps, and the keys and values they leave, against the part-by-part path over the same prompts."""
    from stratum_b200 import StepEntry
    llm, cache = wide, wide.engine.cache
    rng = np.random.default_rng(len(lens) + max(lens))
    toks = [rand_tokens(rng, n + 2, llm.model.vocab) for n in lens]
    out, plan = [], llm.model.resident_steps()
    assert plan is not None
    for on in (True, False):
        llm.model._resident = plan if on else None
        del launches[:]
        slots = _fill(llm, [t[:-2] for t in toks])
        del launches[:]                                      # (a prompt of one token is a step of its own)
        logits = [llm.engine.step([StepEntry(s, [t[i]], [0]) for s, t in zip(slots, toks)]).cpu().numpy() for i in (-2, -1)]
        assert launches == ([len(lens)] * 2 if on else [])
        group, rows = cache.groups[0], cache.page_table_rows(slots, 0)
        kv = [[x[:, row[n // 64], :, n % 64].float().cpu().numpy() for row, n in zip(rows, lens)] for x in (group.k, group.v)]
        out.append((logits, kv))
        for s in slots:
            llm.release(s)
    llm.model._resident = plan
    # Both round the same rows to bfloat16, each sum in its own order: 0.003 to 0.007 of the row's largest logit.  One page left
    # out of the longest row moves it by 0.3 (201 keys) to 0.009 (8,000).
    for a, b in zip(out[0][0], out[1][0]):
        for j in range(len(lens)):
            err = np.max(np.abs(a[j] - b[j])) / np.max(np.abs(b[j]))
            assert err <= 0.01, f"row {j} of {lens[j]} tokens: {err:.4f}"
    for what, a, b in zip("kv", out[0][1], out[1][1]):
        assert_close(np.stack(a), np.stack(b), "bfloat16", what)


def test_steps_on_two_streams(launches):
    """Two models stepped on streams of their own, nothing between the steps that waits: each gives what it gives alone.  (All
    blocks of a launch are resident together or none are, so the two kernels take turns.)"""
    from stratum_b200 import StepEntry, Stratum
    from stratum_b200 import kernels as K
    from stratum_b200.config import LlamaConfig
    rng = np.random.default_rng(12)
    streams, steps, want = [torch.cuda.Stream() for _ in range(2)], [], []
    for seed in (1, 2):
        llm = Stratum.from_random(LlamaConfig.from_dict(WIDE["8B"]), seed=seed, max_tokens=2048, max_seqs=4)
        slots = _fill(llm, [rand_tokens(rng, n, 10000) for n in (300, 700)])
        llm.engine.cache.reserve(slots, [1, 1])
        batch = llm.engine.build_batch([StepEntry(s, [7], [0]) for s in slots])
        want.append(llm.model.forward(batch, llm.engine.cache))
        steps.append((llm, batch))
    torch.cuda.synchronize()
    got = []
    for _ in range(12):
        for i, (llm, batch) in enumerate(steps):
            with torch.cuda.stream(streams[i]):
                got.append((i, llm.model.forward(batch, llm.engine.cache)))
    torch.cuda.synchronize()
    K.check_status()
    assert len(launches) == 26
    assert all(torch.equal(logits, want[i]) for i, logits in got)


EDITS = {
    "one layer's window": lambda m: setattr(m.layers[2].part("mixer"), "window", 24),
    "one layer's scale": lambda m: setattr(m.layers[1].part("mixer"), "scale", 0.02),
    "every layer's scale": lambda m: [setattr(la.part("mixer"), "scale", 0.02) for la in m.layers],
    "one layer's eps": lambda m: setattr(m.layers[3].part("feed_forward_norm"), "eps", 0.5),
    "a part's own forward": lambda m: setattr(m.layers[0].part("feed_forward"), "forward", lambda xn, x, step, emit=None: None),
    "an output bias": lambda m: setattr(m.layers[0].part("mixer").o, "bias", torch.ones(m.hidden, device="cuda")),
}


@pytest.mark.parametrize("edit", sorted(EDITS))
def test_parts_edited_after_the_first_step(model, edit):
    """A step that is launched runs the parts as they are then, not as they were when the model's first step ran."""
    from stratum_b200 import StepEntry
    path, cfg, _ = model
    rng = np.random.default_rng(8)
    toks = [rand_tokens(rng, n + 3, cfg["vocab_size"]) for n in (90, 41)]
    out = []
    for on in (True, False):
        llm = _stratum(path, 1024)
        if not on:
            llm.model._resident, llm.model._resident_asked = None, True
        slots = _fill(llm, [t[:-3] for t in toks])
        step = lambda i: llm.engine.step([StepEntry(s, [t[i]], [0]) for s, t in zip(slots, toks)]).cpu().numpy()   # noqa: E731
        before = step(-3)
        EDITS[edit](llm.model)
        out.append((before, step(-2), step(-1)))
    for a, b in zip(*out):
        assert_close(a, b, "bfloat16", edit)


def _moved(t):
    """The same values, one element behind a 16-byte boundary."""
    out = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape)
    return out.copy_(t)


@pytest.mark.parametrize("which", ["output projection", "down projection", "head", "a norm's gain", "last gain"])
def test_weights_that_no_16_byte_copy_can_read(model, which):
    """A model bound to such tensors runs part by part; nothing is refused."""
    path, cfg, w = model
    llm = _stratum(path, 1024)
    m, layer = llm.model, llm.model.layers[1]
    owner, name = {"output projection": (layer.part("mixer").o, "weight"), "down projection": (layer.part("feed_forward").down, "weight"),
                   "head": (m.head.proj, "weight"), "a norm's gain": (layer.part("feed_forward_norm"), "gain"),
                   "last gain": (m.final_norm, "gain")}[which]
    setattr(owner, name, _moved(getattr(owner, name)))
    t = rand_tokens(np.random.default_rng(9), 40, cfg["vocab_size"])
    slots = _fill(llm, [t[:-1]])
    assert_close(_decode(llm, slots, t[-1:]), plain_logits(cfg, w, t)[-1:], "bfloat16", which)


def test_a_meeting_that_runs_out(model, monkeypatch):
    """Blocks that wait for one more than there are give up after a second: the step ends with an error, no sequence is longer,
    and the next step is right."""
    from stratum_b200 import StepEntry
    from stratum_b200 import kernels as K
    path, cfg, w = model
    llm = _stratum(path, 1024)
    t = rand_tokens(np.random.default_rng(10), 151, cfg["vocab_size"])
    slots = _fill(llm, [t[:150]])
    monkeypatch.setattr(K, "DECODE_LAYERS_ABSENT", 1)
    with pytest.raises(K.KernelError, match="resident decode step"):
        llm.engine.step([StepEntry(slots[0], t[150:], [0])])
    assert llm.engine.length(slots[0]) == 150
    monkeypatch.setattr(K, "DECODE_LAYERS_ABSENT", 0)
    got = llm.engine.step([StepEntry(slots[0], t[150:], [0])]).cpu().numpy()
    assert_close(got, plain_logits(cfg, w, t)[-1:], "bfloat16", "the step behind one that gave up")


def test_sizes_it_refuses():
    """The plan refuses what the launcher's shares and registers do not hold."""
    from stratum_b200 import kernels as K
    dev = torch.device("cuda")
    ok = dict(H=2048, F=8192, vocab=128256, n_q=32, n_kv=8, head_dim=64, device=dev)
    assert K.decode_layers_sizes_ok(**ok)
    for bad in (dict(H=8192), dict(H=2080), dict(F=8200), dict(head_dim=80), dict(n_q=72, n_kv=8), dict(vocab=128257),
                dict(H=128), dict(n_q=128)):
        assert not K.decode_layers_sizes_ok(**dict(ok, **bad)), bad
    assert K.decode_layers_takes(16, 8, 1024, dev) and not K.decode_layers_takes(16, 32, 1024, dev)
