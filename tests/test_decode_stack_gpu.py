"""Decode steps whose layers run as one kernel, against the plain implementation and the kernels of each layer."""
import pytest
import torch

from helpers import assert_close
from plain import qwen3 as plain

pytestmark = pytest.mark.gpu


def config(hidden, ff, nq, nkv, layers=2):
    return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=512, hidden_size=hidden,
                intermediate_size=ff, num_hidden_layers=layers, num_attention_heads=nq, num_key_value_heads=nkv,
                head_dim=128, rope_theta=1000000.0, rms_norm_eps=1e-6, max_position_embeddings=2048,
                tie_word_embeddings=False, use_sliding_window=False, eos_token_id=511)


# groups of 1, 2, 4, 8 query heads; odd and even shares of every product; gate|up of one and of several tiles of rows
MODELS = {"group2": config(256, 1216, 4, 2), "group1": config(320, 2432, 2, 2, 3), "group8": config(576, 1472, 8, 1),
          "group4": config(2560, 9728, 32, 8)}


@pytest.fixture(scope="module")
def engines(tmp_path_factory):
    from grout_b200.engine import Engine
    from grout_b200.weights import write_random_model
    made = {}

    def get(name):
        if name not in made:
            d = str(tmp_path_factory.mktemp(name))
            write_random_model(MODELS[name], 3, d)
            made[name] = (d, Engine.load(d, dtype="bfloat16", max_tokens=8192, max_batch=9, max_seq_len=2048))
        return made[name]
    return get


def played(eng, lens, steps, seed):
    """Prompts of ``lens`` tokens, then ``steps`` decode steps: the tokens, and the decode steps' logits per sequence."""
    g = torch.Generator().manual_seed(seed)
    toks = [torch.randint(0, 511, (n + steps,), generator=g).tolist() for n in lens]
    slots = [eng.open_sequence() for _ in lens]
    for s, t, n in zip(slots, toks, lens):
        eng.step([(s, t[:n])], [[]])
    out = [eng.step([(s, [t[n + i]]) for s, t, n in zip(slots, toks, lens)], [[0]] * len(slots)) for i in range(steps)]
    eng.check()
    for s in slots:
        eng.close_sequence(s)
    return toks, torch.stack(out, dim=1)


@pytest.mark.parametrize("lens", [[1], [63], [64, 5], [127, 128, 700], [1, 62, 190, 191, 192, 333, 1500, 64]], ids=str)
@pytest.mark.parametrize("name", ["group1", "group2", "group8"])
def test_logits_against_the_plain_implementation(engines, name, lens):
    from safetensors import safe_open
    d, eng = engines(name)
    assert eng.model._stack.get(eng.model, eng.cache) is not None
    with safe_open(f"{d}/model.safetensors", "pt") as f:
        w = {k: f.get_tensor(k) for k in f.keys()}
    toks, got = played(eng, lens, 3, 11)
    for i, n in enumerate(lens):
        rows = list(range(n, n + 3))
        assert_close(got[i], plain.logits(w, MODELS[name], toks[i], rows=rows), "bfloat16", f"{name} {lens} sequence {i}")


@pytest.mark.parametrize("lens", [[40], [2000], [100, 900, 3], [300] * 8], ids=str)
def test_as_close_as_layer_by_layer(engines, monkeypatch, lens):
    """The kernel and the kernels of each layer round the same activations to 16 bits and differ in the order of their
    32-bit sums, so their logits differ as two runs of 16-bit activations do: by no more than either's own error, which
    at these sizes is about 1 % of the logits."""
    from grout_b200.engine import stack
    _d, eng = engines("group4")
    _t, got = played(eng, lens, 3, 5)
    monkeypatch.setattr(stack.DecodeStack, "takes", lambda self, step: False)
    eng.graphs.decode_graphs.clear()
    _t, ref = played(eng, lens, 3, 5)
    eng.graphs.decode_graphs.clear()
    err = float((got.double() - ref.double()).norm() / ref.double().norm())
    assert err < 0.02, err


def test_same_bits_every_time(engines):
    _d, eng = engines("group2")
    _t, a = played(eng, [70, 200, 900], 3, 21)
    _t, b = played(eng, [70, 200, 900], 3, 21)
    assert torch.equal(a, b)


@pytest.mark.parametrize("n", [3, 5, 7])
def test_launched_one_by_one_with_any_number_of_rows(engines, n):
    """Without graphs no rows fill a step up to a power of two; sums over the keys may be divided otherwise."""
    _d, eng = engines("group8")
    lens = [33, 64, 129, 5, 700, 64, 1][:n]
    _t, ref = played(eng, lens, 2, 31)
    eng.use_graphs = False
    try:
        _t, got = played(eng, lens, 2, 31)
    finally:
        eng.use_graphs = True
    err = float((got.double() - ref.double()).norm() / ref.double().norm())
    assert err < 0.02, err


def test_other_weights_are_seen(engines):
    """A norm's weight that changes, and a weight that is replaced, reach steps that are launched one by one."""
    _d, eng = engines("group2")
    eng.use_graphs = False
    norm = eng.model.blocks[0].norm2.weight
    before = norm.clone()
    try:
        _t, a = played(eng, [40], 1, 41)
        norm.mul_(0.5)
        _t, b = played(eng, [40], 1, 41)
        norm.copy_(before)
        _t, c = played(eng, [40], 1, 41)
    finally:
        norm.copy_(before)
        eng.use_graphs = True
    assert torch.equal(a, c) and not torch.equal(a, b)


def test_more_rows_than_the_kernel_takes_go_layer_by_layer(engines):
    from grout_b200.engine.batch import make_context
    _d, eng = engines("group2")
    st = eng.model._stack.get(eng.model, eng.cache)
    for n, takes in ((1, True), (8, True), (9, False)):
        assert st.takes(make_context([(0, 0, [1])] * n, None, "cuda")) is takes
    assert not st.takes(make_context([(0, 0, [1, 2])], None, "cuda"))


@pytest.mark.parametrize("change", [dict(head_dim=64), dict(use_sliding_window=True, sliding_window=128, max_window_layers=0)])
def test_other_layers_go_layer_by_layer(change):
    from grout_b200.engine import Engine
    eng = Engine.random(dict(config(256, 1216, 4, 2), **change), 0, max_tokens=512, max_batch=2, max_seq_len=256)
    assert eng.model._stack.get(eng.model, eng.cache) is None


def test_a_replayed_step_sees_norms_that_were_changed_in_place(engines):
    """As the kernels of each layer do: the norms' weights are read where they lie, by captured steps too, also when a
    step that was launched by itself came between."""
    from safetensors import safe_open
    d, eng = engines("group2")
    with safe_open(f"{d}/model.safetensors", "pt") as f:
        w = {k: f.get_tensor(k) for k in f.keys()}
    block = eng.model.blocks[1]
    norms = {"model.layers.1.input_layernorm.weight": block.norm1.weight,
             "model.layers.1.post_attention_layernorm.weight": block.norm2.weight,
             "model.layers.1.self_attn.q_norm.weight": block.mixer.q_norm_w,
             "model.layers.1.self_attn.k_norm.weight": block.mixer.k_norm_w}
    before = {k: t.clone() for k, t in norms.items()}

    def compare(what):
        toks, got = played(eng, [100], 2, 51)
        assert_close(got[0], plain.logits(w, MODELS["group2"], toks[0], rows=[100, 101]), "bfloat16", what)
        return got

    a = compare("captured")
    try:
        for k, t in norms.items():          # every second channel: a common factor would be normalised away again
            t[::2] *= 1.5
            w[k] = t.cpu()
        b = compare("replayed")
        eng.use_graphs = False
        compare("launched by itself")
        eng.use_graphs = True
        c = compare("replayed again")
    finally:
        eng.use_graphs = True
        for k, t in norms.items():
            t.copy_(before[k])
    assert torch.equal(b, c) and not torch.equal(a, b) and torch.equal(a, played(eng, [100], 2, 51)[1])


def test_norms_in_32_bit(engines):
    """bfloat16 weights beside norms that are kept in 32-bit give the same bits as the same norms in bfloat16."""
    _d, eng = engines("group1")
    parts = [n for b in eng.model.blocks for n in (b.norm1, b.norm2)]
    mixers = [b.mixer for b in eng.model.blocks]
    kept = [p.weight for p in parts], [(m.q_norm_w, m.k_norm_w) for m in mixers]
    out = []
    eng.use_graphs = False
    try:
        for wide in (False, True):
            slot = eng.open_sequence()
            eng.step([(slot, list(range(70)))], [[]])
            if wide:
                for p in parts:
                    p.weight = p.weight.float()
                for m in mixers:
                    m.q_norm_w, m.k_norm_w = m.q_norm_w.float(), m.k_norm_w.float()
            out.append(eng.step([(slot, [5])], [[0]]))
            eng.close_sequence(slot)
        eng.check()
    finally:
        eng.use_graphs = True
        for p, t in zip(parts, kept[0]):
            p.weight = t
        for m, (q, k) in zip(mixers, kept[1]):
            m.q_norm_w, m.k_norm_w = q, k
    assert torch.equal(*out)


@pytest.mark.parametrize("graphs", [True, False])
def test_an_engine_made_in_inference_mode(engines, graphs):
    from grout_b200.engine import Engine
    d, eng = engines("group2")
    eng.use_graphs = graphs
    try:
        _t, want = played(eng, [70, 3], 2, 71)
        with torch.inference_mode():
            own = Engine.load(d, dtype="bfloat16", max_tokens=8192, max_batch=9, max_seq_len=2048, use_graphs=graphs)
            _t, got = played(own, [70, 3], 2, 71)
    finally:
        eng.use_graphs = True
    assert torch.equal(got, want)


def one_step(eng, n=300):
    slot = eng.open_sequence()
    eng.step([(slot, list(range(n)))], [[]])
    out = eng.step([(slot, [7])], [[0]])
    eng.close_sequence(slot)
    return out


def test_another_kernels_error_does_not_end_a_step(engines):
    from grout_b200.kernels import ops
    _d, eng = engines("group1")
    want = one_step(eng)
    flag = ops._tc_error_flag(torch.device("cuda:0"))
    flag.fill_(101)
    got = one_step(eng)
    with pytest.raises(ops.KernelError):
        eng.check()
    assert torch.equal(got, want)


def test_a_wait_that_runs_out_voids_the_step_and_not_the_next(engines, monkeypatch):
    """With next to no time to wait, blocks give up on stages, on room in the ring and on one another: they leave, the
    host is told, and the counters are as they were."""
    from grout_b200.kernels import ops
    _d, eng = engines("group1")
    want = one_step(eng)
    st = eng.model.decode_stack(eng.cache)
    monkeypatch.setattr(ops, "DECODE_STACK_WAIT_NS", 1)
    eng.use_graphs = False
    try:
        one_step(eng)
    finally:
        eng.use_graphs = True
    with pytest.raises(ops.KernelError, match="layers' kernel"):
        eng.check()
    assert st.state["sync"].tolist() == [0, 0, 0]
    monkeypatch.setattr(ops, "DECODE_STACK_WAIT_NS", 0)
    assert torch.equal(one_step(eng), want)
    eng.check()


@pytest.fixture
def launches(monkeypatch):
    """The rows of every launch of the kernel (replays do not come here)."""
    from grout_b200.kernels import ops
    rows, run = [], ops.decode_stack

    def counted(state, res, pending, **kw):
        out = run(state, res, pending, **kw)
        rows.append(out.shape[0])
        return out
    monkeypatch.setattr(ops, "decode_stack", counted)
    return rows


def test_the_kernel_is_what_runs(engines, launches):
    _d, eng = engines("group4")
    eng.graphs.decode_graphs.clear()
    played(eng, [100, 900, 3], 2, 5)
    assert launches == [4, 4]              # the warm-up and the capture of one bucket, whose second step is a replay
    eng.use_graphs = False
    try:
        played(eng, [100, 900, 3], 2, 5)
        assert launches == [4, 4, 3, 3]
        played(eng, [9] * 9, 1, 5)
        assert launches == [4, 4, 3, 3]    # nine rows go layer by layer
    finally:
        eng.use_graphs = True


def test_a_replaced_weight_is_seen(engines, launches):
    from safetensors import safe_open
    d, eng = engines("group2")
    with safe_open(f"{d}/model.safetensors", "pt") as f:
        w = {k: f.get_tensor(k) for k in f.keys()}
    lin = eng.model.blocks[0].mixer.o
    before = lin.weight
    eng.use_graphs = False
    try:
        lin.weight = before.flip(0).contiguous()
        w["model.layers.0.self_attn.o_proj.weight"] = lin.weight.cpu()
        toks, got = played(eng, [100], 2, 81)
    finally:
        lin.weight = before
        eng.use_graphs = True
    assert launches == [1, 1]
    assert_close(got[0], plain.logits(w, MODELS["group2"], toks[0], rows=[100, 101]), "bfloat16", "another o projection")


MODELS["many_kv"] = config(256, 1216, 32, 32)


@pytest.mark.parametrize("lens", [[5, 500, 64, 127, 300], [1, 62, 190, 191, 192, 333, 508, 64]], ids=str)
def test_two_units_of_attention_in_a_block(engines, launches, lens):
    """More (sequence, kv head) pairs than blocks."""
    from safetensors import safe_open
    d, eng = engines("many_kv")
    with safe_open(f"{d}/model.safetensors", "pt") as f:
        w = {k: f.get_tensor(k) for k in f.keys()}
    eng.use_graphs = False
    try:
        toks, got = played(eng, lens, 3, 13)
    finally:
        eng.use_graphs = True
    assert launches[-3:] == [len(lens)] * 3          # (a prompt of one token is a decode step of its own)
    for i, n in enumerate(lens):
        want = plain.logits(w, MODELS["many_kv"], toks[i], rows=list(range(n, n + 3)))
        assert_close(got[i], want, "bfloat16", f"{lens} sequence {i}")


@pytest.mark.parametrize("nq,nkv,lens", [(8, 1, [6100]), (32, 32, [35000]), (16, 8, [33000, 20000, 34000, 200])], ids=str)
def test_long_sequences(launches, nq, nkv, lens):
    """The most splits of a head's keys (96 tiles in 32), more tiles in a block (137) than it keeps the pages of, and long
    sequences beside a short one; keys and values are random.  Against the kernels of each layer, as above."""
    from grout_b200.engine import Engine, stack
    eng = Engine.random(dict(config(256, 1216, nq, nkv), max_position_embeddings=40960), 4, max_batch=4, max_seq_len=40960,
                        max_tokens=sum(lens) + 64 * 8, use_graphs=False)
    g = torch.Generator(device="cuda").manual_seed(1)
    for i in range(2):
        view = eng.cache.view(i)
        view.k_pages.normal_(generator=g)
        view.v_pages.normal_(generator=g)
    slots = [eng.open_sequence() for _ in lens]
    for s, n in zip(slots, lens):
        eng.cache.reserve(s, n + 1)
        eng.cache.length[s] = n

    def step():
        out = eng.step([(s, [7 + s]) for s in slots], [[0]] * len(slots))
        for s, n in zip(slots, lens):
            eng.cache.length[s] = n
        return out.double()

    got = step()
    assert launches == [len(lens)]
    with pytest.MonkeyPatch.context() as m:
        m.setattr(stack.DecodeStack, "takes", lambda self, step: False)
        want = step()
    eng.check()
    assert launches == [len(lens)]
    err = float((got - want).norm() / want.norm())
    assert err < 0.02, err
