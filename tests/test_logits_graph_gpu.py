"""Decode steps of `forward_cb` through captured graphs: against the same steps run eagerly, over batch sizes that are padded,
contexts that cross a width of the block table, pools that grow, rows given by the caller, and results that outlive later steps."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(monkeypatch, path, graph, name="tiny-llama", **kw):
    import xfastertransformer_b200 as xft
    from xfastertransformer_b200.tools.synthetic import preset, write_synthetic_checkpoint
    from xfastertransformer_b200.utils.flags import Env
    monkeypatch.setenv("XFT_CUDA_GRAPH", str(int(graph)))
    Env.get().reload()
    if not list(path.iterdir()):
        write_synthetic_checkpoint(str(path), preset(name), seed=3)
    m = xft.AutoModel.from_pretrained(str(path), dtype="bf16", **kw)
    monkeypatch.delenv("XFT_CUDA_GRAPH")
    Env.get().reload()
    return m


def _same(a, b):
    """Split counts may differ with the width of the table: sums in another order, then the bf16 roundings of two layers."""
    assert a.shape == b.shape
    assert (a - b).norm() <= 2.0 ** -6 * b.norm(), ((a - b).norm() / b.norm()).item()


# widths of the table change at 8 and 16 blocks of 64; 3 and 9 rows are padded to 4 and 12
@pytest.mark.parametrize("lens", [[1], [5, 300, 508], [60] * 9, [1018, 2, 511]])
@pytest.mark.parametrize("name", ["tiny-llama", "tiny-dagezen"])
def test_steps_match_eager(lens, name, monkeypatch, tmp_path):
    g = torch.Generator().manual_seed(len(lens))
    eager, graph = (_model(monkeypatch, tmp_path, on, name) for on in (False, True))
    vocab = graph.model.cfg.vocab_size
    prompts = [torch.randint(0, vocab, (n,), generator=g).tolist() for n in lens]
    steps = [torch.randint(0, vocab, (len(lens),), generator=g).tolist() for _ in range(9)]
    outs = []
    for m in (eager, graph):
        ids = m.set_input_cb(prompts, None, 1100).tolist()
        out = [m.forward_cb()]
        for t in steps:
            m.set_input_cb(t, ids)
            out.append(m.forward_cb())
        outs.append(out)
        m.free_seqs(ids)
    assert graph.model.runner.graph_launches >= 3 and eager.model.runner.graph_launches == 0
    for a, b in zip(outs[1], outs[0]):                       # read after all steps: no result is overwritten
        _same(a, b)


def test_growing_pools_rows_and_mixed_steps(monkeypatch, tmp_path):
    eager, graph = (_model(monkeypatch, tmp_path, on) for on in (False, True))
    outs = []
    for m in (eager, graph):
        out = []
        a = m.set_input_cb([[7, 8, 9]], None, 200).tolist()
        out.append(m.forward_cb())
        for i in range(4):
            m.set_input_cb([11 + i], a)
            out.append(m.forward_cb())
        b = m.set_input_cb([list(range(500))], None, 3000).tolist()          # the pools move: graphs are made again
        out.append(m.forward_cb())
        for i in range(4):
            m.set_input_cb([21 + i], a, rows=[[0]])
            out.append(m.forward_cb())
        m.set_input_cb([31, 32], a + b, rows=[[], [0]])                       # a step without one sequence's logits
        out.append(m.forward_cb())
        m.set_input_cb([33, 34], a + b)
        m.set_input_cb([[1, 2, 3, 4]], None, 64, append=True)                 # a prompt beside running sequences
        out.append(m.forward_cb())
        outs.append(out)
    for x, y in zip(outs[1], outs[0]):
        _same(x, y)


def test_steps_on_another_stream(monkeypatch, tmp_path):
    eager, graph = (_model(monkeypatch, tmp_path, on) for on in (False, True))
    side, outs = torch.cuda.Stream(), []
    for m in (eager, graph):
        ids, out = m.set_input_cb([[3, 1, 4, 1, 5]], None, 100).tolist(), []
        m.forward_cb()
        for i in range(8):
            here = side if i % 3 == 2 else torch.cuda.default_stream()
            here.wait_stream(torch.cuda.default_stream())
            with torch.cuda.stream(here):
                m.set_input_cb([40 + i], ids)
                out.append(m.forward_cb())
            torch.cuda.default_stream().wait_stream(here)
        torch.cuda.synchronize()
        outs.append(out)
    for x, y in zip(outs[1], outs[0]):
        _same(x, y)


def test_streams_that_nobody_orders(monkeypatch, tmp_path):
    """Prompts, eager and captured steps, greedy steps and a pool that moves, each on another stream than the one before, without an
    event between them: the engine puts its passes in order, whose scratch and caches are the same memory."""
    eager, graph = (_model(monkeypatch, tmp_path, on) for on in (False, True))
    streams = [torch.cuda.default_stream(), torch.cuda.Stream(), torch.cuda.Stream()]
    outs = []
    for m, mixed in ((eager, False), (graph, True)):
        out, ids, turn = [], [], 0

        def call(fn):
            nonlocal turn
            turn += 1
            with torch.cuda.stream(streams[turn % 3 if mixed else 0]):
                out.append(fn())

        def start(prompt, room):
            ids.extend(m.set_input_cb([prompt], None, room).tolist())
            return m.forward_cb()

        def step(tokens, greedy=False):
            m.set_input_cb(tokens, ids, greedy=greedy)
            return m.forward_cb_greedy() if greedy else m.forward_cb()
        call(lambda: start(list(range(5, 400)), 600))
        for i in range(7):
            call(lambda: step([40 + i]))
        call(lambda: start(list(range(300)), 6000))
        for i in range(7):
            call(lambda: step([60 + i, 80 + i]))
        for i in range(4):
            call(lambda: step([90 + i, 95 + i], greedy=True))
        for i in range(4):
            call(lambda: step([70 + i, 50 + i]))
        torch.cuda.synchronize()
        outs.append(out)
    assert graph.model.runner.graph_launches >= 8
    for x, y in zip(outs[1], outs[0]):
        if x.is_floating_point():
            _same(x, y)


@pytest.mark.parametrize("lens", [[150], [500, 40], [700, 1100]])
@pytest.mark.parametrize("name", ["tiny-llama", "latent"])
def test_captured_steps_cut_attention_as_eager_ones(lens, name, monkeypatch, tmp_path):
    """Batches that are not padded: the table of a captured step is wider, its launches are otherwise those of an eager step, so the
    logits are the same bits."""
    from xfastertransformer_b200.tools import synthetic
    if name == "latent":
        from xfastertransformer_b200.config import ModelConfig
        cfg = ModelConfig(model_type="deepseek_moe", num_layer=2, hidden_size=512, head_num=8, kv_head_num=8, size_per_head=128, inter_size=1024,
                          vocab_size=1024, max_pos_seq_len=4096, q_lora_rank=256, kv_lora_rank=512, qk_nope_head_dim=128, qk_rope_head_dim=64,
                          v_head_dim=128, moe_intermediate_size=256, first_k_dense_replace=1, dense_experts=1, sparse_experts=16,
                          routed_scaling_factor=2.5, topk_method="noaux_tc", n_group=4, topk_group=2, num_experts_per_tok=4, norm_topk_prob=True,
                          scoring_func="sigmoid", activation_type="silu", weight_data_type="bf16", start_id=0, end_id=1)
        write = synthetic.write_synthetic_checkpoint
        monkeypatch.setattr(synthetic, "preset", lambda _: cfg)
        monkeypatch.setattr(synthetic, "write_synthetic_checkpoint", lambda p, c, seed: write(p, c, seed=seed, dtype="bf16", std=0.05))
    eager, graph = (_model(monkeypatch, tmp_path, on, name, kv_cache_dtype="bf16") for on in (False, True))
    g = torch.Generator().manual_seed(sum(lens))
    prompts = [torch.randint(2, 1000, (n,), generator=g).tolist() for n in lens]
    outs = []
    for m in (eager, graph):
        ids, out = m.set_input_cb(prompts, None, 1300).tolist(), []
        m.forward_cb()
        for i in range(6):
            m.set_input_cb([10 + i, 20 + i][:len(lens)], ids)
            out.append(m.forward_cb())
        outs.append(out)
    assert graph.model.runner.graph_launches >= 3
    assert all(torch.equal(a, b) for a, b in zip(*outs))
