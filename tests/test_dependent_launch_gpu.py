"""Steps whose kernels are all waiting in the stream, so that each is launched while the one before it runs: the same bits as one
after the other, whatever the scratch buffers hold from the step before."""
import pytest

pytestmark = pytest.mark.gpu

HOLD = 4_000_000          # clocks (about 2 ms) that the stream is held: longer than the host takes to launch a step
LENGTHS = [272, 170, 1300, 1210, 60, 2, 1]


def _llama(tmp):
    from helpers import SMALL_E, random_prompt, random_weights, write_model_dir
    d = write_model_dir(str(tmp / "m"), SMALL_E, random_weights(SMALL_E, seed=2, norm_std=0.1, std=0.03), "bfloat16")
    return d, [random_prompt(SMALL_E, n, i) for i, n in enumerate(LENGTHS)]


def _drawn_tuzapel(tmp):
    """A general-size latent, wide values, experts chosen one, five and two at a time."""
    from helpers import write_model_dir
    from tuzapel_helpers import prompt, random_config, random_weights
    cfg = random_config(220, True)
    d = write_model_dir(str(tmp / "m"), cfg, random_weights(cfg, 6), "bfloat16")
    return d, [prompt(cfg, n, i) for i, n in enumerate(LENGTHS)]


def _other(name):
    def make(tmp):
        import importlib
        h = importlib.import_module(name + "_helpers")
        d, cfg = h.make_model(tmp, "C", seed=7)[:2]
        return d, [h.prompt(cfg, n, i) for i, n in enumerate(LENGTHS)]
    return make


MODELS = {"llama": _llama, "tuzapel_drawn": _drawn_tuzapel,
          **{n: _other(n) for n in ("notirax", "luzinex", "rabapel", "ledinex", "takavik", "tuzapel")}}


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("model", list(MODELS))
def test_steps_behind_a_held_stream(model, dtype, tmp_path):
    import torch
    from mlxforge_b200.csrc import ops
    from mlxforge_b200.engine.replay import make_runner
    from mlxforge_b200.engine.step import StepEntry
    d, prompts = MODELS[model](tmp_path)

    def run(dependent):
        old = ops.set_dependent_launch(dependent)
        try:
            runner = make_runner(d, dtype, 8192, max_seqs=8)
            outs = []

            def step(entries):
                if dependent:
                    torch.cuda._sleep(HOLD)
                outs.append(runner.step(entries).clone())

            for p in prompts:                                   # whole prompts, one after another
                s = runner.cache.open_sequence()
                step([StepEntry(s, p, list(range(len(p))))])
                runner.cache.close(s)
            seqs = [runner.cache.open_sequence() for _ in prompts]
            step([StepEntry(s, p[:len(p) // 2 + 1], [len(p) // 2]) for s, p in zip(seqs, prompts)])
            step([StepEntry(s, p[len(p) // 2 + 1:], [0]) for s, p in zip(seqs, prompts) if len(p) > 2])       # portions
            for i in range(5):                                  # decoding: eager, captured, replayed
                step([StepEntry(s, [p[i % len(p)]], [0]) for s, p in zip(seqs, prompts)])
            torch.cuda.synchronize()
            ops.check_kernel_status()
            return outs
        finally:
            ops.set_dependent_launch(old)

    want = run(False)
    for _ in range(2):
        for i, (a, b) in enumerate(zip(want, run(True))):
            assert not bool(torch.isnan(a).any()) and torch.equal(a, b), i
