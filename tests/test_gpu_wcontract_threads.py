"""Products with MPOs of different bonds, and so of different shared memory, from several threads at once."""
import threading

import pytest
import torch

import tnpy_gb300.kernels as K

pytestmark = pytest.mark.gpu


def test_products_of_different_mpo_bonds_in_threads():
    bonds, failed = [17, 24, 32, 20], []
    start = threading.Barrier(len(bonds))

    def work(dl):
        try:
            g = torch.Generator(device="cuda").manual_seed(dl)
            rand = lambda *s: torch.randn(*s, generator=g, dtype=torch.float64, device="cuda")
            L, R, x, w = rand(8, dl, 8), rand(8, dl, 8), rand(8, 2, 8), rand(dl, dl, 2, 2)
            with torch.cuda.stream(torch.cuda.Stream()):
                ref = K.matvec1(L, w, R, x)
                torch.cuda.current_stream().synchronize()
                start.wait()
                for _ in range(1500):
                    y = K.matvec1(L, w, R, x)
                torch.cuda.current_stream().synchronize()
                assert torch.equal(y, ref)
        except Exception as e:  # reported by the test's own thread
            failed.append((dl, repr(e)))

    threads = [threading.Thread(target=work, args=(dl,)) for dl in bonds]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
