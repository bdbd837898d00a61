"""ocipProximityIndx of several threads on one context: every call gets its own template's place."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", ["PATH_AUTO", "PATH_PLAIN"])
def test_threads_get_their_own_best_match(ocip, ctx, path):
    ctx.make_current()
    rng = np.random.default_rng(8)
    S = rng.integers(0, 256, (160, 220), dtype=np.uint8)
    places = [(5, 9), (100, 31), (150, 120), (40, 77)]
    T = [S[y:y + 24, x:x + 24].copy() for x, y in places]
    source, templates = ocip.Image(S), [ocip.Image(t) for t in T]
    for r in [source] + templates:
        r.send()
    ctx.set_path(getattr(ocip, path))
    want = [(0, 0.0, x + 12, y + 12) for x, y in places]
    wrong = []

    def run(k):
        for _ in range(100):
            got = ocip.proximity_index("SqrDistance", "MinIndx", source, templates[k])
            if got != want[k]:
                wrong.append((k, got))

    try:
        for k in range(4):
            assert ocip.proximity_index("SqrDistance", "MinIndx", source, templates[k]) == want[k]
        threads = [threading.Thread(target=run, args=(k,)) for k in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        ctx.set_path(ocip.PATH_PLAIN)
    for r in [source] + templates:
        r.release()
    assert not wrong, wrong[:4]
