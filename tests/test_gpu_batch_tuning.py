"""vb_batch_set_tuning's CTAs per SM are of 256 threads in both precisions."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [1, 2])
def test_ctas_per_sm_count_256_threads(ctas):
    import torch

    from verona_b200.batch import Batch, riemann_problems

    specs, prims = riemann_problems(3, n1d=2, n2d=2, n1d_range=(2048, 4096), n2d_range=(256, 512), gamma=5.0 / 3.0)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for precision, threads in (("fp64", 256), ("fp32", 128)):
        b = Batch(specs, 5.0 / 3.0, rk=3, precision=precision, riemann="hllc", n_iter=50, tol=1e-12, floor=1e-8)
        b.set_tuning(0, ctas)
        for i, P in enumerate(prims):
            b.load_prims(i, P)
        b.step(1)
        assert b.check() == 0 and b.tuning["grid"] * threads == ctas * sms * 256
        b.close()
