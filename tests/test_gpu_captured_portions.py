"""Prompt portions behind a long cache as serving runs them: captured steps, padded tokens and sequences, a context class in which the
CTAs of a cluster share a tile's pages and the tiles are listed; against the plain model."""
import numpy as np
import pytest

import helpers
from test_gpu_schedules import _tolerance, real_heads                               # noqa: F401

pytestmark = pytest.mark.gpu


def _run(folder, tmp_path, steps, requests):
    from oracle_engine_b200.engine.engine import Engine
    eng = Engine.from_pretrained(folder, dtype="bfloat16", max_tokens=4096)
    out = helpers.TraceRunner(eng, tmp_path / "run").run(steps)
    eng.check_device_errors()
    eng.cache.check()
    at, got = {i: 0 for i in requests}, {i: {} for i in requests}
    for s in steps:
        row = 0
        for e in s["entries"]:
            for w in e["want"]:
                got[e["id"]][at[e["id"]] + w] = out[s["step"]][row]
                row += 1
            at[e["id"]] += len(e["tokens"])
    return eng, got


def _compare(plain, requests, got):
    for i, toks in requests.items():
        want = plain.logits(toks).cpu().numpy()
        tol = _tolerance(want)
        for pos, row in got[i].items():
            err = np.abs(row - want[pos]).max()
            assert err < tol, f"request {i} position {pos}: {err} (tolerance {tol})"


def _captured(eng):
    return {key[:4] for key, g in eng.stepper._token_graphs.items() if g.graph is not None}


def test_portions_beside_decoding_sequences(real_heads, tmp_path):               # noqa: F811
    """Three sequences padded to four, 72 to 102 tokens padded to 128: two decode, one of them past 768 tokens, and one brings portions of
    unequal length over its own cache.  The first such step runs directly, the second is captured, the others are replayed."""
    from oracle_engine_b200.csrc import ops_tc
    folder, plain = real_heads
    portions = (70, 61, 90, 100, 65, 77)
    lens = {"long": 900 + len(portions), "short": 40 + len(portions), "portions": sum(portions)}
    requests = {i: helpers.random_tokens(n, 512, 50 + n) for i, n in lens.items()}
    entry = lambda i, a, n, want: {"id": i, "tokens": requests[i][a:a + n], "want": want}              # noqa: E731
    steps = [{"step": 0, "entries": [entry("long", 0, 900, [899])], "end": []}, {"step": 1, "entries": [entry("short", 0, 40, [39])], "end": []}]
    at = 0
    for k, n in enumerate(portions):
        steps.append({"step": 2 + k, "entries": [entry("long", 900 + k, 1, [0]), entry("short", 40 + k, 1, [0]), entry("portions", at, n, [0, n // 2, n - 1])], "end": []})
        at += n
    steps[-1]["end"] = list(requests)
    eng, got = _run(folder, tmp_path, steps, requests)
    assert (128, 4, 64, 1) in _captured(eng) and ops_tc.prompt_cluster(128, 4, 3, 8, 1, sm_count=148) == 2
    _compare(plain, requests, got)


@pytest.mark.parametrize("portions,key,cluster", [((40, 33, 64, 51, 60), (64, 1, 64, 1), 8), ((100, 65, 128, 90, 127), (128, 1, 64, 1), 4),
                                                  ((200, 129, 256, 150), (256, 1, 64, 1), 2)])
def test_portions_of_one_sequence_behind_a_long_cache(real_heads, tmp_path, portions, key, cluster):           # noqa: F811
    """800 tokens, then portions that clusters of 8, 4 and 2 CTAs walk, captured and replayed; up to 64 places of each are wanted."""
    from oracle_engine_b200.csrc import ops_tc
    folder, plain = real_heads
    requests = {"one": helpers.random_tokens(800 + sum(portions), 512, 7 + len(portions) + portions[0])}
    steps = [{"step": 0, "entries": [{"id": "one", "tokens": requests["one"][:800], "want": [0, 799]}], "end": []}]
    at = 800
    for k, n in enumerate(portions):
        steps.append({"step": 1 + k, "entries": [{"id": "one", "tokens": requests["one"][at:at + n], "want": list(range(0, n, (n + 63) // 64))}], "end": []})
        at += n
    steps[-1]["end"] = ["one"]
    eng, got = _run(folder, tmp_path, steps, requests)
    assert key in _captured(eng) and ops_tc.prompt_cluster(key[0], 1, 3, 8, 1, sm_count=148) == cluster
    _compare(plain, requests, got)
