"""Concurrent callers, a context each: row counts and lengths whose launches
of one kernel take different amounts of shared memory."""
import threading

import numpy as np
import pytest

import golaypair_gb300 as gp

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,first,second", [
    (gp.GP_PSD_FP64, (45, 2**19), (45, 300)), (gp.GP_PSD_FP64, (500, 4096), (2, 64)),
    (gp.GP_PSD_TC_GUARDED, (33, 3000), (47, 3000)), (gp.GP_PSD_TC_GUARDED, (113, 700), (127, 700)),
])
def test_threads_filter_at_once(mode, first, second):
    go = threading.Barrier(2)
    errors = []

    def work(L, n, calls):
        try:
            rng = np.random.default_rng(n + L)
            x = torch.from_numpy(rng.choice(np.array([-2, 0, 2], dtype=np.int8), size=(n, L))).cuda()
            masks = [torch.zeros((n + 31) // 32, dtype=torch.int32, device="cuda") for _ in range(2)]
            torch.cuda.synchronize()
            with gp.Context(0) as ctx:
                order = 2 * L
                ctx.psd_filter_device(x.data_ptr(), n, L, order, 0, mode, masks[0].data_ptr(), stats=True)
                go.wait()
                for _ in range(calls):
                    ctx.psd_filter_device(x.data_ptr(), n, L, order, 0, mode, masks[1].data_ptr())
                ctx.psd_filter_device(x.data_ptr(), n, L, order, 0, mode, masks[1].data_ptr(), stats=True)
            assert torch.equal(*masks)
        except Exception as e:
            errors.append(e)
            go.abort()

    threads = [threading.Thread(target=work, args=(*case, 4000)) for case in (first, second)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
