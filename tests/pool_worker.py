"""Run in a process of its own by test_gpu_scratch_pool.py, so that its contexts are the device's
only ones: scratch taken from several threads and streams while contexts come and go."""
import threading

import numpy as np

from renzoku_b200 import rzk


def threads():
    import torch
    rng = np.random.default_rng(1)
    jobs = []
    for k in range(4):
        m = torch.from_numpy(rng.gamma(0.3, 1.0, (700 + 100 * k, 40 + k, 3)).astype(np.float32)).cuda()
        jobs.append((m, [a.clone() for a in rzk.ClusterBuilderCuda().alphas(m)],
                     rzk.ClusterBuilderCuda().cluster_by_sampling(m, 30, 5)))
    torch.cuda.synchronize()
    bad = []

    def work(m, alphas, clusters):
        try:
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                for _ in range(60):
                    got = rzk.ClusterBuilderCuda().alphas(m)
                    again = rzk.ClusterBuilderCuda().cluster_by_sampling(m, 30, 5)
                    st.synchronize()
                    if not (all(torch.equal(a, b) for a, b in zip(got, alphas))
                            and all(np.array_equal(a, b) for a, b in zip(again, clusters))):
                        bad.append("values")
        except Exception as e:   # reported by the main thread
            bad.append(repr(e))

    ts = [threading.Thread(target=work, args=j) for j in jobs]
    for t in ts:
        t.start()
    n = 0
    while any(t.is_alive() for t in ts):
        rzk.Context(0).close()
        n += 1
    for t in ts:
        t.join()
    assert not bad and n > 10, (bad, n)


if __name__ == "__main__":
    threads()
    print("worker ok")
