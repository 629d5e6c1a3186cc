"""Router calls of different lengths from several threads.  Needs a B200.

The limit on dynamic shared memory belongs to the kernel, not to the launch: a call with short rows must not lower it
between another thread's setting and its launch."""

import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_short_and_long_rows_at_once(native_lib):
    from h3_optimizations_b200 import ops

    errors, outputs = [], {}

    def work(tiles):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                gen = torch.Generator(device="cuda").manual_seed(tiles)
                q, k = (torch.randint(-3, 4, (1, 2, n, 128), generator=gen, device="cuda").double() for n in (16, tiles))
                call = lambda: ops.route_topk(q, k, q_start=0, q_stop=16, kv_start=0, kv_stop=tiles, retained=tiles // 3)
                first = call()
                for _ in range(3000):
                    again = call()
                torch.cuda.current_stream().synchronize()
                outputs[tiles] = torch.equal(first, again)
        except Exception as error:  # noqa: BLE001 - reported by the main thread
            errors.append("%d tiles: %s" % (tiles, error))

    threads = [threading.Thread(target=work, args=(tiles,)) for tiles in (16, 2300, 17, 2200)]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    assert not errors, errors[0]
    assert all(outputs.values()) and len(outputs) == 4
