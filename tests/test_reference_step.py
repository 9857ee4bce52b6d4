"""The fused training step of the reference architecture (csrc/reference_step.cu, small_optimizer_kernel)
against the same engine running operator by operator on CUDA cores."""
import ctypes as C

import numpy as np
import pytest
import torch

from helpers import relative
from turbogpt_b200 import bridge
from turbogpt_b200.bridge import Config, ConfigEx, Native

pytestmark = pytest.mark.gpu

# Tile edges: one padded sequence; sequences that straddle a warp's 16 rows; a last tile with fewer sequences;
# a sequence longer than a warp and one that fills a tile; the shipped experiment; more tiles than SMs (two
# rounds: gradients accumulate across tiles); the deepest model that fits.
SHAPES = [(1, 2, 3), (2, 5, 7), (4, 4, 16), (3, 16, 9), (2, 33, 5), (2, 128, 3), (4, 4, 2880), (8, 8, 2001), (16, 7, 41)]
NAMES = ["x", "normed1", "qkv", "attended", "middle", "normed2", "activated"]


def engine_pair(depth, context, batch, scheduled):
    rng = np.random.default_rng(depth * 1000 + context)
    data = rng.integers(32, 127, 4096 + context, dtype=np.uint8)
    engines = []
    for flags in (0, bridge.FLAG_NO_TENSOR_CORES):
        ex = ConfigEx.reference(Config(depth=depth, context=context, batch=batch), flags=flags)
        engine = Native(ex)
        engine.set_weights(bridge.initialize_weights(ex))
        if scheduled:
            engine.set_onecycle(100)
        engine.set_data(data)
        engines.append(engine)
    return engines, bridge.parameter_layout(ex)


@pytest.mark.parametrize("depth,context,batch", SHAPES)
def test_step_matches_the_operator_path(depth, context, batch):
    (fused, plain), layout = engine_pair(depth, context, batch, True)
    with fused, plain:
        before = fused.weights()
        for engine in (fused, plain):
            engine.train(1)
        # Losses: those of the step's own logits (BF16 values of final_normed and the head's high halves) in 64 bits.  FP32
        # losses of 4 to 8 carry two ulps of 2^-21 each way; sums in another order flip at most one row's logit by an ulp.
        losses, plain_losses = fused.training_losses(1)[0], plain.training_losses(1)[0]
        offset, rows, cols = layout[-1]
        head = (before[offset:offset + rows * cols].view(np.uint32) & np.uint32(0xffff0000)).view(np.float32).reshape(rows, cols)
        normed = fused.activation(-1, "final_normed").astype(np.float64)
        logits = torch.from_numpy((normed @ head.T).astype(np.float32)).bfloat16().double()
        _, targets = fused.sample(0)
        exact = torch.nn.functional.cross_entropy(logits, torch.from_numpy(targets.ravel().astype(np.int64)), reduction="none")
        ulp = 2 ** -8 * float(logits.abs().max())
        np.testing.assert_allclose(losses, exact.reshape(batch, context).mean(0).numpy(), rtol=0, atol=2 ** -20 + ulp / batch)
        # Against the operator path: both round the logits to BF16, of activations that may differ by a flipped rounding.
        np.testing.assert_allclose(losses, plain_losses, rtol=0, atol=ulp)
        for name in NAMES:
            for layer in (0, depth - 1):
                assert relative(fused.activation(layer, name), plain.activation(layer, name)) <= 5e-3, (layer, name)
        assert relative(fused.activation(-1, "final_normed"), plain.activation(-1, "final_normed")) <= 5e-3
        # After one step the momentum is a fixed multiple of the gradient: the reference's per-tensor bound.
        (m, v, step), (pm, pv, _) = fused.optimizer_state(), plain.optimizer_state()
        assert step == 1
        for offset, rows, cols in layout:
            part = slice(offset, offset + rows * max(cols, 1))
            assert relative(m[part], pm[part]) <= 0.02, (offset, rows, cols)
            if np.any(pv[part]):
                assert relative(v[part], pv[part]) <= 0.04, (offset, rows, cols)
        # The update itself: the operator path's optimizer on the gradient this step used (the first step's sign-like
        # AdamW update and Muon's null directions amplify the gradients' own differences, so those are kept out), with the
        # reference's bounds for AdamW and Muon (tests/verify.py).
        plain.set_weights(before)
        rates = bridge.StepRates()
        bridge.load_library().tg_onecycle_point(C.byref(bridge.OneCycle(100)), 0, C.byref(rates))
        plain.optimizer_test(m / np.float32(1 - rates.momentum))
        expected, got = plain.weights(), fused.weights()
        for offset, rows, cols in layout:
            part = slice(offset, offset + rows * max(cols, 1))
            if cols and rows != 256:
                assert relative(got[part] - before[part], expected[part] - before[part]) <= 0.04, (offset, rows, cols)
            else:
                np.testing.assert_allclose(got[part], expected[part], atol=2e-6, rtol=2e-5)


@pytest.mark.parametrize("depth,context,batch,row_tiles,rounds,helpers,overlap", [
    (2, 80, 2, 5, 1, 0, 0), (2, 96, 150, 6, 2, 0, 0), (3, 100, 4, 7, 1, 0, 0),
    (3, 16, 149 * 2 + 1, 3, 1, 1, 1), (16, 32, 3, 2, 1, 1, 1), (16, 48, 3, 3, 1, 1, 0),
    (16, 32, 150, 2, 2, 1, 1), (16, 16, 500, 2, 2, 1, 1), (12, 16, 800, 3, 2, 1, 1)])  # gradients added to the first tile's
def test_tiles_with_helpers_and_without(depth, context, batch, row_tiles, rounds, helpers, overlap):
    """The same bounds as everywhere."""
    ex, plan = ConfigEx.reference(Config(depth=depth, context=context, batch=batch)), (C.c_int32 * 5)()
    assert bridge.load_library().tg_ex_reference_step_plan(C.byref(ex), 148, plan) == 0
    rows, tiles, blocks, *form = plan
    assert (rows // 16, -(-tiles // blocks), *form) == (row_tiles, rounds, helpers, overlap)
    test_step_matches_the_operator_path(depth, context, batch)


def test_no_bit_of_a_token_depends_on_the_tile_it_is_in():
    """15 sequences over 15, 8, 5, 3, 2 and 1 blocks: 1, 2 and 3 row tiles of a block, with helpers, 5 and 8 without, in one
    or two rounds.  Activations are a token's own; and as every byte occurs once, so is its embedding's gradient.
    (60 batches: sums in another order flip about one BF16 rounding in 30000.)"""
    rng = np.random.default_rng(11)
    inputs = [(rng.permutation(256)[:240].astype(np.uint8).reshape(15, 16), rng.integers(0, 256, (15, 16), dtype=np.uint8))
              for _ in range(60)]
    results = []
    for blocks in (15, 8, 5, 3, 2, 1):
        ex = ConfigEx.reference(Config(depth=4, context=16, batch=15, blocks=blocks, clip=0))
        w, outputs = bridge.initialize_weights(ex) * 8, []  # branches of the residual stream's own size
        with Native(ex) as engine:
            for x, y in inputs:
                engine.set_weights(w)
                engine.train_batch(x, y)
                outputs += [engine.activation(-1, "final_x"), engine.optimizer_state()[0][:4096]]
        results.append(outputs)
    assert np.count_nonzero(results[0][-1]) > 3000
    for other in results[1:]:
        assert sum(np.count_nonzero(a != b) for a, b in zip(results[0], other)) == 0


@pytest.mark.parametrize("depth,context,batch", [(4, 4, 16), (2, 5, 7), (8, 8, 2001)])
def test_graph_direct_and_streamed_steps_are_the_same(depth, context, batch):
    """Replayed graphs, direct launches and steps fed from host bytes leave bit-identical weights."""
    rng = np.random.default_rng(1)
    data = rng.integers(32, 127, 4096, dtype=np.uint8)
    results = []
    for flags, streamed in ((0, False), (bridge.FLAG_NO_GRAPH, False), (0, True)):
        ex = ConfigEx.reference(Config(depth=depth, context=context, batch=batch), flags=flags)
        with Native(ex) as engine:
            engine.set_weights(bridge.initialize_weights(ex))
            engine.set_data(data)
            if streamed:
                losses = np.stack([engine.train_batch(*engine.sample(step)) for step in range(30)])
            else:
                engine.train(19)
                first = engine.training_losses(19)
                engine.train(11)
                losses = np.concatenate([first, engine.training_losses(11)])
            results.append((losses, engine.weights(), engine.optimizer_state()[0]))
    for other in results[1:]:
        for a, b in zip(results[0], other):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("depth,context,batch", [(2, 5, 7), (3, 16, 9), (2, 3, 2001)])  # padded rows, none, several tiles a block
@pytest.mark.parametrize("byte,occurs", [(0, False), (200, True)])
def test_an_infinite_embedding_reaches_what_it_reaches_operator_by_operator(depth, context, batch, byte, occurs):
    """The embedding of one byte value overflows.  Where no token reads it, nothing changes; otherwise the gradients that
    turn NaN are those of the operator path: other bytes' embeddings keep theirs."""
    (fused, plain), layout = engine_pair(depth, context, batch, False)
    rng = np.random.default_rng(3)
    x, y = rng.integers(32, 127, (batch, context), dtype=np.uint8), rng.integers(32, 127, (batch, context), dtype=np.uint8)
    if occurs:
        x[::3, context // 2] = byte
    with fused, plain:
        w = fused.weights()
        w[byte * 16:byte * 16 + 16] = np.inf
        moments = []
        for engine in (fused, plain):
            engine.set_weights(w)
            engine.train_batch(x, y)
            moments.append(engine.optimizer_state()[0])
        a, b = moments
        assert occurs or np.isfinite(a).all()
        np.testing.assert_array_equal(np.isfinite(a[:4096]), np.isfinite(b[:4096]))
        assert np.isfinite(b[:4096]).sum() > 2048  # the embedding's gradients are worth comparing
        finite = np.isfinite(b[:4096])
        assert relative(a[:4096][finite], b[:4096][finite]) <= 0.02  # the reference's per-tensor bound


def test_a_profiled_engine_times_every_family():
    """The fused step has no families: a profiled engine runs the operators, and their times are told apart."""
    ex = ConfigEx.reference(Config(depth=2, context=4, batch=16), flags=bridge.FLAG_PROFILE)
    with Native(ex) as engine:
        engine.set_weights(bridge.initialize_weights(ex))
        engine.set_data(np.random.default_rng(0).integers(32, 127, 4096, dtype=np.uint8))
        engine.train(2)
        engine.training_losses(2)
        families = engine.profile()
    missing = {name for name, (milliseconds, launches) in families.items() if not (milliseconds > 0 and launches > 0)}
    assert missing == {"gradient_exchange"}  # one GPU exchanges nothing
