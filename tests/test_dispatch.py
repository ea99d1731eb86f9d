"""Which kernel a call is given to: the rules of parts/gemm_dispatch.py and parts/attention_dispatch.py, with the
launchers replaced by recorders (no GPU needed)."""
import types

import pytest
import torch


@pytest.fixture
def recorded(monkeypatch):
    from stratum_b200 import kernels as K
    calls = []

    def recorder(name):
        def f(*args, **kwargs):
            calls.append((name, args, kwargs))
        return f

    for name in ("gemm_skinny", "gemm_tc", "linear_simple", "swiglu", "attention_simple", "attention_stream",
                 "attention_mma", "attention_tc", "attention_tile"):
        monkeypatch.setattr(K, name, recorder(name))
    return calls


def _xw(rows, n, k, dtype=torch.bfloat16):
    return torch.zeros(rows, k, dtype=dtype), torch.zeros(n, k, dtype=dtype), torch.zeros(rows, n, dtype=dtype)


def test_matrix_product_rules(recorded):
    from stratum_b200.parts import gemm_dispatch as G
    small, large = (4096, 4096), (28672, 4096)                  # 16.8 M and 117 M weights
    assert small[0] * small[1] < G.STREAMK_MIN_WEIGHTS <= large[0] * large[1]
    for rows, shape, want in ((1, small, "gemm_skinny"), (G.SKINNY_MAX_ROWS, small, "gemm_skinny"),
                              (G.SKINNY_MAX_ROWS + 1, small, "gemm_tc"), (1, large, "gemm_tc"),
                              (2048, small, "gemm_tc")):
        recorded.clear()
        x, w, out = _xw(rows, *shape)
        G.run(x, w, None, out, G.STORE)
        assert [c[0] for c in recorded] == [want], (rows, shape)
    # float32 is the true 32-bit path whatever the shape; so is a row pitch that no 16-byte copy can start on
    for x, w, out in (_xw(8, 4096, 4096, torch.float32), _xw(8, 64, 20)):
        recorded.clear()
        G.run(x, w, None, out, G.ADD_TO_F32)
        assert [c[0] for c in recorded] == ["linear_simple"]
    # SwiGLU without a tensor-core kernel: the product, then the activation
    recorded.clear()
    x, w, _ = _xw(3, 64, 20)
    G.run(x, w, None, torch.zeros(3, 32, dtype=torch.bfloat16), G.SWIGLU)
    assert [c[0] for c in recorded] == ["linear_simple", "swiglu"]


def _attention_call(recorded, dtype, head_dim, n_heads, n_kv, n_tokens, all_single):
    from stratum_b200.parts import attention_dispatch as A
    recorded.clear()
    att = types.SimpleNamespace(head_dim=head_dim, n_heads=n_heads, n_kv_heads=n_kv, window=0, scale=1.0,
                                runtime=types.SimpleNamespace(scratch=lambda name, n, dt: torch.zeros(n, dtype=dt)))
    width = (n_heads + 2 * n_kv) * head_dim
    qkv = torch.zeros(n_tokens, width, dtype=dtype)
    cache = types.SimpleNamespace(k=None, v=None, block_table=None)
    step = types.SimpleNamespace(all_single=all_single, n_tokens=n_tokens, max_len=300, token_pos=None,
                                 token_seq=None, query_blocks=lambda n: None)
    A.run(att, qkv, cache, step, torch.zeros(n_tokens, n_heads * head_dim, dtype=dtype))
    assert len(recorded) == 1
    return recorded[0]


def test_attention_rules(recorded):
    bf, f32 = torch.bfloat16, torch.float32
    name, args, _ = _attention_call(recorded, f32, 128, 32, 8, 80, True)
    assert name == "attention_simple" and args[-1] is True           # told that no two tokens share a sequence's pages
    assert _attention_call(recorded, f32, 128, 32, 8, 80, False)[1][-1] is False
    assert _attention_call(recorded, bf, 256, 4, 2, 8, True)[0] == "attention_simple"        # head size above 128
    name, _, kw = _attention_call(recorded, bf, 128, 32, 8, 8, True)
    assert name == "attention_stream" and kw["late_trigger"] is True
    assert _attention_call(recorded, bf, 64, 8, 2, 2, True)[2]["late_trigger"] is False     # one or two sequences
    # heads of 64: whole pages per warp once an SM gets more than a few pages (here 5 pages a sequence and kv head)
    assert _attention_call(recorded, bf, 64, 8, 2, 100, True)[2]["whole_pages"] is False    # 1,000 pages
    assert _attention_call(recorded, bf, 64, 32, 8, 64, True)[2]["whole_pages"] is True     # 2,560 pages
    assert _attention_call(recorded, bf, 128, 32, 8, 64, True)[2]["whole_pages"] is False
    assert _attention_call(recorded, bf, 80, 6, 2, 8, True)[0] == "attention_mma"            # head size 80
    assert _attention_call(recorded, bf, 128, 12, 1, 8, True)[0] == "attention_mma"          # 12 heads per kv head
    assert _attention_call(recorded, bf, 128, 32, 8, 300, False)[0] == "attention_tc"
    assert _attention_call(recorded, bf, 128, 3, 1, 300, False)[0] == "attention_tile"       # 128 % 3 != 0
    assert _attention_call(recorded, bf, 96, 8, 2, 300, False)[0] == "attention_tile"


def test_extra_epilogue_rules(recorded, monkeypatch):
    """Where a product carries more than its basic epilogue: rows of a handed-over norm and the query/key/value
    epilogue go to the tensor-core kernel or are refused; a Handover is honoured where the product's tiles fill the SMs
    (hands_over); prompt attention gets query tiles of 256 rows."""
    from stratum_b200 import kernels as K
    from stratum_b200.parts import gemm_dispatch as G
    from stratum_b200.parts.base import Handover, NormedRows, Runtime
    from stratum_b200.parts.linear import ADD_TO_F32, STORE, Linear
    small = (4096, 4096)
    x, w, out = _xw(4, *small)
    assert not G.takes_tensor_cores(x, w, extras=False) and G.takes_tensor_cores(x, w, extras=True)
    G.run(x, w, None, out, G.STORE, extra=object())               # few rows, small matrix: still the tensor cores
    assert [c[0] for c in recorded] == ["gemm_tc"]
    with pytest.raises(K.KernelError, match="only the tensor-core kernel"):
        G.run(*_xw(4, 64, 20)[:2], None, torch.zeros(4, 64, dtype=torch.bfloat16), G.STORE, extra=object())
    # Linear: the residual add honours a Handover only with enough rows
    monkeypatch.setattr(K, "_need", lambda *a, **k: None)        # (the tensors of this test live on the host)
    monkeypatch.setattr(K, "gemm_tc", lambda *a, **k: (recorded.append(("gemm_tc", a, k)), 7)[1])
    rt = types.SimpleNamespace(dtype=torch.bfloat16, device="cpu",
                               empty=lambda *shape, dtype=torch.bfloat16: torch.zeros(shape, dtype=dtype))
    lin = Linear(rt, torch.zeros(4096, 4096, dtype=torch.bfloat16))
    gain = torch.ones(4096)
    assert not G.hands_over(768, 4096) and G.hands_over(769, 4096)          # 48 and 64 tiles of 256 x 256
    assert not G.hands_over(1024, 2048) and G.hands_over(2048, 2048)
    monkeypatch.setattr(G, "HANDOVER_MIN_TILES", 1)
    for rows, honoured in ((G.HANDOVER_MIN_ROWS - 1, False), (G.HANDOVER_MIN_ROWS, True)):
        recorded.clear()
        ask = Handover(gain, 4096, 1e-5)
        lin(torch.zeros(rows, 4096, dtype=torch.bfloat16), out=torch.zeros(rows, 4096), mode=ADD_TO_F32, emit=ask)
        assert (ask.result is not None) == honoured
        assert [c[0] for c in recorded] == ["gemm_tc"]
        assert recorded[0][1][4] == (K.EPI_ADD_F32_EMIT if honoured else K.EPI_ADD_F32)
        if honoured:
            r = ask.result
            assert isinstance(r, NormedRows) and r.parts == 7 and r.x.shape == (rows, 4096) and r.size == 4096
            # and the product behind the norm takes them as rows to be scaled
            recorded.clear()
            lin(r, mode=STORE)
            assert recorded[0][1][4] == K.EPI_STORE and recorded[0][1][5].c.norm_parts == 7
    # prompt attention: a CTA's query tile is 256 rows (2 x 128 / group size tokens), 128 when asked for
    from stratum_b200.parts import attention_dispatch as A
    sizes = []
    att = types.SimpleNamespace(head_dim=128, n_heads=32, n_kv_heads=8, window=0, scale=1.0, runtime=None)
    step = types.SimpleNamespace(all_single=False, n_tokens=300, max_len=300, token_pos=None, token_seq=None,
                                 query_blocks=lambda n: sizes.append(n))
    cache = types.SimpleNamespace(k=None, v=None, block_table=None)
    for env, tokens in ((None, 64), ("1", 32)):
        if env:
            monkeypatch.setenv("STRATUM_ATTENTION_HALVES", env)
        recorded.clear()
        A.run(att, torch.zeros(300, 48 * 128, dtype=torch.bfloat16), cache, step, torch.zeros(300, 4096, dtype=torch.bfloat16))
        assert recorded[0][0] == "attention_tc" and sizes[-1] == tokens


def test_shared_memory_is_opted_into_at_every_launch():
    """The opt-in belongs to the device that is current when it is made, and may fail once: no launcher keeps its result for
    the life of the process."""
    import glob
    import os
    import re
    import stratum_b200
    sources = glob.glob(os.path.join(os.path.dirname(stratum_b200.__file__), "csrc", "*.cu*"))
    assert len(sources) > 20
    for path in sources:
        with open(path) as f:
            assert not re.search(r"static\b[^;{}]*=[^;{}]*cudaFuncSetAttribute", f.read()), path


def test_resident_steps_ask_for_a_block_per_sm(monkeypatch):
    """What the resident kernel's launcher refuses its plan refuses too: devices of more SMs than its tables hold."""
    from stratum_b200 import kernels as K
    for sms, takes in ((132, True), (148, True), (160, True), (161, False), (192, False)):
        monkeypatch.setattr(K, "sm_count", lambda device, n=sms: n)
        assert K.decode_layers_sizes_ok(4096, 14336, 128256, 32, 8, 128, None) == takes


def _step_of(rows, width):
    tables = {0: torch.zeros(rows, width, dtype=torch.int32)}
    return types.SimpleNamespace(n_tokens=rows, block_tables=tables, token_ids=torch.zeros(rows, dtype=torch.int32))


def test_resident_steps_go_the_same_way_launched_and_replayed(monkeypatch):
    """The rule sees a launched step's own rows and pages and a replay's padded ones: it must not tell them apart, up to the
    kernel's limit on pages (1,007 a block) and beyond it."""
    from stratum_b200 import kernels as K
    from stratum_b200.engine.graphs import padded_rows, width_bucket
    from stratum_b200.engine.resident import ResidentSteps
    monkeypatch.setattr(K, "sm_count", lambda device: 148)
    seen = set()
    for heads in ((32, 8, 128), (32, 32, 128), (32, 8, 64), (16, 16, 64)):
        att = types.SimpleNamespace(n_heads=heads[0], n_kv_heads=heads[1], head_dim=heads[2], hidden=4096, window=0)
        decoder = types.SimpleNamespace(att=att)
        for rows in range(1, 17):
            for width in (1, 3, 8, 9, 16, 17, 257, 291, 292, 512, 580, 582, 583, 1000, 1024, 1025):
                launched = ResidentSteps.takes(decoder, _step_of(rows, width))
                assert launched == ResidentSteps.takes(decoder, _step_of(padded_rows(rows), width_bucket(width)))
                # what it takes, the launcher takes
                assert not launched or K.decode_layers_takes(rows, heads[1], width, None)
                seen.add(launched)
    assert seen == {True, False}


# (rows, pages of the table, kv heads, head size, width, heads * size): what was measured on 148 SMs, us part by part / resident
MEASURED_STEPS = [
    ((1, 4, 8, 64, 2048, 2048), True),        # 856 / 639
    ((8, 16, 8, 64, 2048, 2048), True),       # 965 / 810
    ((8, 128, 8, 64, 2048, 2048), True),      # 1,261 / 1,128
    ((8, 512, 8, 64, 2048, 2048), False),     # 2,185 / 2,209
    ((16, 4, 8, 64, 2048, 2048), True),       # 968 / 908
    ((16, 16, 8, 64, 2048, 2048), True),      # 1,059 / 1,032
    ((16, 512, 8, 64, 2048, 2048), False),    # 3,465 / 3,608
    ((8, 64, 8, 128, 4096, 4096), True),      # 1,902 / 1,773
    ((8, 512, 8, 128, 4096, 4096), True),     # 4,048 / 3,918
    ((16, 4, 8, 128, 4096, 4096), False),     # 1,772 / 1,825
    ((16, 64, 8, 128, 4096, 4096), False),    # 2,137 / 2,187
    ((8, 128, 32, 128, 4096, 4096), True),    # 3,805 / 3,660
    ((16, 8, 32, 128, 4096, 4096), False),    # 1,880 / 1,970
    ((8, 64, 32, 64, 2048, 2048), True),      # 1,258 / 1,132
    ((8, 512, 32, 64, 2048, 2048), False),    # 5,754 / 6,466
    ((1, 64, 4, 64, 2048, 2048), True),       # 856 / 753
    ((8, 64, 8, 64, 1024, 1024), True),       # 605 / 593
    ((8, 128, 8, 64, 1024, 1024), False),     # 816 / 857
    ((8, 16, 2, 128, 1536, 1536), False),     # 4 rows: 829 / 854
    ((4, 128, 4, 64, 2048, 2048), True),      # 907 / 802
    ((1, 16, 1, 128, 2048, 1024), True),      # 1,013 / 685
    ((1, 128, 1, 128, 2048, 1024), False),    # 1,122 / 1,849
    ((4, 128, 1, 128, 2048, 1024), False),    # 881 / 1,087
    ((2, 128, 2, 128, 1536, 1536), False),    # 926 / 1,145
    ((8, 64, 12, 64, 768, 768), False),       # 417 / 452
    ((8, 8, 12, 64, 768, 768), True),         # 322 / 292
    ((8, 16, 2, 64, 512, 512), False),        # 106 / 119
    ((1, 512, 2, 64, 512, 512), False),       # 157 / 221
]


@pytest.mark.parametrize("sizes,pays", MEASURED_STEPS, ids=lambda v: str(v))
def test_resident_steps_where_they_are_shorter(monkeypatch, sizes, pays):
    from stratum_b200 import kernels as K
    from stratum_b200.engine.resident import ResidentSteps
    monkeypatch.setattr(K, "sm_count", lambda device: 148)
    rows, width, n_kv, head_dim, hidden, heads_width = sizes
    att = types.SimpleNamespace(n_heads=heads_width // head_dim, n_kv_heads=n_kv, head_dim=head_dim, hidden=hidden,
                                window=0)
    assert ResidentSteps.takes(types.SimpleNamespace(att=att), _step_of(rows, width)) == pays


def test_resident_parameters_are_described_alike(monkeypatch):
    """The struct and its mirror are of one size, and a launch with another is refused."""
    import ctypes
    from stratum_b200 import kernels as K
    monkeypatch.setattr(K, "_decode_layers_checked", False)
    assert K._decode_layers_fn() is not None and K._decode_layers_checked
    monkeypatch.setattr(K, "_decode_layers_checked", False)
    monkeypatch.setattr(K, "_DecodeLayers", ctypes.c_char * 64)
    with pytest.raises(K.KernelError):
        K._decode_layers_fn()


@pytest.mark.skipif(torch.cuda.is_available(), reason="the parameters name no memory: only a machine that cannot launch asks this")
def test_resident_launcher_refuses():
    """The launcher's own questions, one broken at a time, before it calls CUDA at all."""
    import ctypes
    from stratum_b200 import kernels as K
    SHAPE, ALIGN, LIMIT = -2, -3, -4
    f = K._decode_layers_fn()

    def status(blocks=148, layer=None, **over):
        p = K._DecodeLayers()
        for name, kind in p._fields_:
            if kind is ctypes.c_void_p:
                setattr(p, name, 4096)
        for n in range(4):
            for name, _ in K._DecodeLayer._fields_:
                setattr(p.layer[n], name, 4096)
        sizes = dict(bt_stride=64, n_layers=4, M=8, H=4096, F=14336, n_q=32, n_kv=8, D=128, n_pairs=64, vocab=128256,
                     eps=1e-5, scale=0.1)
        for name, v in dict(sizes, **over).items():
            setattr(p, name, v)
        for name, v in (layer or {}).items():
            setattr(p.layer[3], name, v)
        return f(ctypes.addressof(p), blocks, None)

    assert status() > 0                                    # (no device: a CUDA error, not a refusal)
    assert status(M=0) == 0
    for want, cases in ((LIMIT, [dict(M=17), dict(n_layers=97), dict(blocks=161), dict(bt_stride=0), dict(bt_stride=3000), dict(M=1, bt_stride=20000)]),
                        (SHAPE, [dict(n_layers=0), dict(blocks=0), dict(D=80), dict(n_kv=5), dict(n_kv=0), dict(n_q=72), dict(n_pairs=65),
                                 dict(n_pairs=-1), dict(H=4160), dict(H=8192), dict(H=256), dict(F=14400), dict(F=128), dict(n_q=64),
                                 dict(vocab=1001), dict(vocab=200), dict(vocab=-2), dict(x=None), dict(w_head=None),
                                 dict(logits=None), dict(rope=None), dict(status=None), dict(counters=None), dict(part_ml=None),
                                 dict(layer=dict(w_o=None)), dict(layer=dict(v=None))]),
                        (ALIGN, [dict(x=4104), dict(w_head=4098), dict(rope=4104), dict(layer=dict(k=4098)),
                                 dict(layer=dict(gain_next=4100))])):
        for c in cases:
            assert status(**c) == want, c
    assert status(vocab=0, w_head=None, logits=None) > 0   # a step that wants no logits
    assert status(n_pairs=0, rope=None) > 0
