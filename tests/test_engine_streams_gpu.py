"""The engine's extra streams (weight gradients, mean loss, padded output weights) against the same step on one stream."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(hidden, batch, overlap, vocab=65):
    from cme213_final_project_b200.config import ModelConfig, OptimConfig, RunConfig
    from cme213_final_project_b200.models.engine import NativeEngine
    # GELU: no pre-activation that rounding takes across zero switches a gradient on or off
    cfg = ModelConfig(vocab_size=vocab, seq_len=32, hidden=hidden, heads=4, ff=2 * hidden, batch_size=batch, activation="gelu")
    eng = NativeEngine(cfg, OptimConfig(), RunConfig(), device="cuda", seed=3)
    eng.set_overlap(overlap)
    # weights of the size that keeps a layer's output at its input's: with the small uniform start the softmax is flat, and
    # what reaches d ln1 through it is a difference of nearly equal sums, all rounding
    g = torch.Generator().manual_seed(7)
    flat = torch.zeros(eng.layout.total)
    for s in eng.layout.specs:
        v = torch.randn(s.numel, generator=g) * {"weight": hidden ** -0.5, "embed": 1.0}.get(s.kind, 0.1)
        flat[s.offset:s.offset + s.numel] = v + (1.0 if s.kind == "ln_gamma" else 0.0)
    eng.set_params(flat.to(torch.bfloat16).float())
    return eng, cfg


def _batches(cfg, n):
    g = torch.Generator().manual_seed(5)
    draw = lambda: torch.randint(0, 65, (cfg.tokens_per_step,), generator=g, dtype=torch.int32).cuda()      # noqa: E731
    return [draw() for _ in range(n)], [draw() for _ in range(n)]


@pytest.mark.parametrize("micro", [1, 3])
@pytest.mark.parametrize("hidden", [32, 64, 96, 200, 256])
def test_streams_give_the_step_of_one_stream(hidden, micro):
    from cme213_final_project_b200.config import OptimConfig
    from cme213_final_project_b200.models.reference import ReferenceModel
    runs = []
    for overlap in (False, True, True):
        eng, cfg = _engine(hidden, 8, overlap)
        xs, ys = _batches(cfg, micro)
        for _ in range(3):
            eng.train_step(xs, ys)
        runs.append((eng.grads.clone(), eng.loss_dev.clone()))
    for g, loss in runs[1:]:
        assert torch.equal(g, runs[0][0]) and torch.equal(loss, runs[0][1])
    ref = ReferenceModel(cfg, OptimConfig(), device="cpu", dtype=torch.float64, seed=3, layout=eng.layout)
    ref.params.data.copy_(eng.master.cpu())
    want = torch.zeros(eng.layout.total, dtype=torch.float64)
    for x, y in zip(xs, ys):
        ref.zero_grad()
        ref.forward(x.cpu(), y.cpu())
        ref.backward()
        want += ref.grads.double() / micro
    for name in ("ln1_gamma", "ln1_beta", "tok_embed", "pos_embed"):          # what d ln1 goes into
        s = eng.layout.by_name[name]
        sl = slice(s.offset, s.offset + s.numel)
        # a handful of bf16 roundings (2^-9 each) of values that enter as sums of the same size
        assert ((eng.grads[sl].cpu().double() - want[sl]).norm() / want[sl].norm()).item() < 3e-2


@pytest.mark.parametrize("hidden,batch", [(256, 8), (512, 304)])
def test_fences_of_a_captured_backward(hidden, batch):
    """Buckets that another stream reads behind a fence, captured as ``forward`` + ``backward``: the third stream is no part of the
    graph before its first product, or at all where a weight gradient is more than 10 GFLOP (the second size)."""
    eng, cfg = _engine(hidden, batch, True)
    (x,), (y,) = _batches(cfg, 1)
    buckets = eng.layout.coalesced_buckets(1)
    reader, copy, errors = torch.cuda.Stream(), torch.empty_like(eng.grads), []

    def ready(b):
        try:
            eng.fence(reader)
            with torch.cuda.stream(reader):
                copy[b.start:b.end].copy_(eng.grads[b.start:b.end])
        except Exception as e:                              # (an exception does not leave the native call)
            errors.append(e)

    def step():
        eng.forward(x, y)
        eng.backward(ready, buckets)
        torch.cuda.current_stream().wait_stream(reader)

    step()
    torch.cuda.synchronize()
    assert len(buckets) > 2 and torch.equal(copy, eng.grads)
    want = copy.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    assert not errors
    for _ in range(3):
        copy.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(copy, want)


@pytest.mark.parametrize("seq,batch", [(64, 128), (64, 304), (128, 8), (256, 64)])
def test_layers_that_share_buffers_between_streams(seq, batch):
    """Four blocks (a buffer that one block's weight gradients still read is overwritten by the next block's chain only behind a
    wait; the dQ scratch alternates between blocks), several steps in flight: with half of the weight gradients on the third
    stream (9.7 GFLOP each with 64 tokens, 1.2 with 128) and with the loss alone there (23 and 19 GFLOP)."""
    from cme213_final_project_b200.config import ModelConfig, OptimConfig, RunConfig
    from cme213_final_project_b200.models.engine import NativeEngine
    cfg = ModelConfig(mode="gpt", vocab_size=65, seq_len=seq, hidden=384, heads=6, ff=1536, layers=4, batch_size=batch,
                      activation="gelu", causal=True, head_layout="split", tied_embeddings=True, final_layernorm=True, init="normal")
    xs, ys = _batches(cfg, 4)
    runs = []
    for overlap in (False, True, True):
        eng = NativeEngine(cfg, OptimConfig(), RunConfig(), device="cuda", seed=3)
        eng.set_overlap(overlap)
        steps = []
        for x, y in zip(xs, ys):                            # (nothing waits for a step before the next is enqueued)
            eng.train_step([x], [y])
            steps.append((eng.grads.clone(), eng.loss_dev.clone()))
        eng.train_step(xs, ys)                              # four micro-batches
        steps.append((eng.grads.clone(), eng.loss_dev.clone()))
        runs.append(steps)
    for steps in runs[1:]:
        for (g, loss), (want, want_loss) in zip(steps, runs[0]):
            assert torch.equal(loss, want_loss)
            if seq <= 64:                                   # every sum in a fixed order
                assert torch.equal(g, want)
            else:
                # the parts of dQ are added in arrival order: some of its bf16 values come out one unit (2^-8) off, which
                # goes on through the blocks below; per tensor far less than all of them at once
                for s in eng.layout.specs:
                    a, b = g[s.offset:s.offset + s.numel].float(), want[s.offset:s.offset + s.numel].float()
                    assert ((a - b).norm() / b.norm()).item() < 2.0 ** -8, s.name


@pytest.mark.parametrize("vocab", [65, 4096, 12288])
def test_loss_beside_short_and_before_long_products_of_the_head(vocab):
    """The mean loss and its publication run beside the backward pass or, where the head's products are more than 10 GFLOP (the
    largest vocabulary), before it: the same loss, whichever way it is read, and the same gradients."""
    runs = []
    for overlap in (False, True):
        eng, cfg = _engine(256, 64, overlap, vocab)
        xs, ys = _batches(cfg, 3)
        seen = []
        for i in range(3):
            eng.seq_expected += 1
            eng.train_step(xs[:i + 1], ys[:i + 1])          # one to three micro-batches
            seen.append(eng.wait_loss())
            assert seen[-1] == eng.read_loss()
        runs.append((seen, eng.grads.clone()))
    assert runs[0][0] == runs[1][0] and torch.equal(runs[0][1], runs[1][1])
