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
