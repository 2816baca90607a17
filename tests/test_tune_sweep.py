"""What the autotuner times for each knob of the multiply: the call that the knob
governs, and nothing for a knob without effect (no GPU: a context and a scheme that
record their calls)."""
import torch

from kunpbfv_b200 import tune


class _Ctx:
    N, log_n, q_count, p_count, dnum, L = 8, 3, 2, 1, 1, 1

    def __init__(self):
        self.knobs, self.calls = {"fuse_q2r_pairs": 1}, []

    def tune_get(self, knob):
        return self.knobs.get(knob, 0)

    def tune_set(self, knob, value):
        self.knobs[knob] = value

    def zeros(self, *shape):
        return torch.zeros(shape, dtype=torch.int64)

    def bconv_q_to_r(self, x):
        self.calls.append("bconv")
        return x + 1


class _Scheme:
    def __init__(self, ctx):
        self.context = ctx

    def mult_relin(self, a, b, out):
        self.context.calls.append("mult_relin")


def test_every_sweep_times_what_its_knob_governs(monkeypatch):
    ctx = _Ctx()
    timed = {}

    def sweep(c, knob, values, run, out, want, reps):
        ctx.calls.clear()
        run()
        timed[knob] = set(ctx.calls)
        return {v: float(i) for i, v in enumerate(values)}

    monkeypatch.setattr(tune, "_sweep", sweep)
    monkeypatch.setattr(tune, "_random_pairs", lambda c, n, seed: torch.zeros(n, 2, c.q_count, c.N, dtype=torch.int64))
    monkeypatch.setattr(torch.cuda, "synchronize", lambda: None)
    got = tune.tune_pipeline(_Scheme(ctx), pairs=8)
    assert timed.pop("bconv_cpt") == {"bconv"}, "governs the standalone conversions only"
    assert "fuse_q2r_pairs" not in timed, "has no effect"
    assert timed and all(c == {"mult_relin"} for c in timed.values())
    assert got["fuse_q2r_pairs"] == 1 and got["bconv_cpt"] == tune.BCONV_CPT[0]
    assert "fuse_q2r_pairs" not in tune.PIPELINE_CHOICES
