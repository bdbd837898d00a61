"""Index reductions of several threads on one context, each with a program of its own: every call
gets its own image's answer."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(9, 5), (640, 480)])
def test_threads_get_their_own_answers(ocip, ctx, W, H):
    ctx.make_current()
    images, programs, want = [], [], []
    for k in range(4):
        S = np.zeros((H, W), np.float32)
        x, y = (3 + 2 * k) % W, k % H
        S[y, x] = k + 1
        images.append(ocip.Image(S))
        images[-1].send()
        programs.append(ocip.prepare_statistics(images[-1]))
        want.append((0, float(k + 1), x, y))
        assert ocip.index_reduce("MaxIndx", programs[k], images[k]) == want[k]
    wrong = []

    def run(k):
        for _ in range(200):
            got = ocip.index_reduce("MaxIndx", programs[k], images[k])
            if got != want[k]:
                wrong.append((k, got))

    threads = [threading.Thread(target=run, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for r in programs + images:
        r.release()
    assert not wrong, wrong[:4]
