"""The allocation-free level-2 assembly in single takes no shared scratch: calls
from several threads on streams of their own, each with other matrices, give
what they give one after another, bit for bit."""
import threading

import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests.test_zzzz_no_alloc import _col, _pch

pytestmark = pytest.mark.gpu


def test_concurrent_single_calls():
    from top_gpu_on_matlab_b200._lib import TOP_F32, TOP_OK, lib
    m = O.Model(np.ones((24, 40, 32), bool), control=20000)
    m.apply_optcase(1)
    L0, L1 = m.level(0), m.level(1)
    nE, nCh = L1.elementUpwardMap.shape
    up, P, mu = _col(L1.elementUpwardMap, torch.int32), _col(_pch(4), torch.float32), _col(m.mapUniqueKes(), torch.int32)
    fr, fx = (_col(a, torch.float32) for a in m.uniqueKes())
    nU = m.uniqueKes()[0].shape[1]
    E = _col(0.05 + np.random.default_rng(31).random(L0.numElements), torch.float32)
    workers = 4
    K0 = [_col(L0.Ke * (1 + w), torch.float32) for w in range(workers)]
    out = [torch.empty(576 * nE, dtype=torch.float32, device="cuda") for _ in range(workers)]

    def call(w, stream):
        return lib().top_assemble_ks_level2_noalloc(out[w].data_ptr(), up.data_ptr(), E.data_ptr(), K0[w].data_ptr(), P.data_ptr(), mu.data_ptr(),
                                                    fr.data_ptr(), fx.data_ptr(), nE, nCh, E.numel(), nU, TOP_F32, stream)

    ref = []
    for w in range(workers):
        assert call(w, None) == TOP_OK
        ref.append(out[w].clone())
    streams = [torch.cuda.Stream() for _ in range(workers)]
    torch.cuda.synchronize()
    wrong = []

    def work(w):
        for _ in range(40):
            if call(w, streams[w].cuda_stream) != TOP_OK:
                wrong.append(w)
                return
            with torch.cuda.stream(streams[w]):
                if not torch.equal(out[w], ref[w]):
                    wrong.append(w)

    threads = [threading.Thread(target=work, args=(w,)) for w in range(workers)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
