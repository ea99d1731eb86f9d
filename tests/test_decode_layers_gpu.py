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
def wherever_it_can(monkeypatch):
    """These tests are of the kernel: it takes every step it can run, not only those that are shorter in it."""
    from stratum_b200.engine import resident
    monkeypatch.setattr(resident, "pays", lambda *a: True)


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
def test_against_the_oracle(model, lens):
    path, cfg, w = model
    llm = _stratum(path, sum(n + 128 for n in lens))
    rng = np.random.default_rng(len(lens))
    steps = 3
    toks = [rand_tokens(rng, n + steps, cfg["vocab_size"]) for n in lens]
    slots = _fill(llm, [t[:n] for t, n in zip(toks, lens)])
    got = [_decode(llm, slots, [t[n + i] for t, n in zip(toks, lens)]) for i in range(steps)]
    assert llm.model.resident_steps() is not None
    for j, (t, n) in enumerate(zip(toks, lens)):
        ref = plain_logits(cfg, w, t)
        assert_close(np.stack([g[j] for g in got]), ref[n:], "bfloat16", f"row {j} of {n} tokens")


def test_window_and_rows_alone(model):
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


def test_steps_it_leaves_alone(model):
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
    _decode(llm, slots[3:], [t[19] for t in toks[3:]])
    got = _decode(llm, slots, [t[20] for t in toks])
    assert_close(got[:3], np.stack([r[20] for r in ref]), "bfloat16", "seventeen rows")
    for s in slots:
        llm.release(s)
    a, b = _fill(llm, [t[:19] for t in toks[:2]]), _fill(llm, [t[:19] for t in toks[:2]])
    replayed = _decode(llm, a, [t[19] for t in toks[:2]])
    launched = llm.engine.step([StepEntry(s, [t[19]], [0]) for s, t in zip(b, toks)]).cpu().numpy()
    assert np.array_equal(replayed, launched)


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
    """The launcher refuses what its shares and registers do not hold; the plan asks the same questions."""
    from stratum_b200 import kernels as K
    dev = torch.device("cuda")
    ok = dict(H=2048, F=8192, vocab=128256, n_q=32, n_kv=8, head_dim=64, device=dev)
    assert K.decode_layers_sizes_ok(**ok)
    for bad in (dict(H=8192), dict(H=2080), dict(F=8200), dict(head_dim=80), dict(n_q=72, n_kv=8), dict(vocab=128257),
                dict(H=128), dict(n_q=128)):
        assert not K.decode_layers_sizes_ok(**dict(ok, **bad)), bad
    assert K.decode_layers_takes(16, 8, 1024, dev) and not K.decode_layers_takes(16, 32, 1024, dev)
