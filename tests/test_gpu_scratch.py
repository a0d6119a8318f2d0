"""Entry points that allocate scratch per call (chfsi_zgemm_cn, chfsi_hegv_dev)
from several threads on several streams: the pool they share hands each call its
own memory."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("m,n,k", [(20, 20, 2945), (261, 77, 23847)])
def test_concurrent_calls_have_their_own_scratch(chfsi, m, n, k):
    rng = np.random.default_rng(5)
    sets = []
    for _ in range(4):
        a = torch.from_numpy(rng.standard_normal((m, k)) + 1j * rng.standard_normal((m, k))).cuda()
        b = torch.from_numpy(rng.standard_normal((n, k)) + 1j * rng.standard_normal((n, k))).cuda()
        sets.append((a, b, a.conj() @ b.T))
    torch.cuda.synchronize()
    bad = []

    def work(i):
        a, b, ref = sets[i]
        st = torch.cuda.Stream()
        c = torch.empty((m, n), dtype=torch.complex128, device="cuda")
        torch.cuda.synchronize()
        for _ in range(10):
            chfsi.zgemm_cn(a.data_ptr(), k, b.data_ptr(), k, m, n, k, c.data_ptr(), st.cuda_stream)
            # two FP64 sums of k terms: each within sqrt(k) 2^-52 of |a||b| ~ 2k
            if float((c - ref).abs().max()) > 4 * k ** 0.5 * 2.0 ** -52 * 2 * k:
                bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
