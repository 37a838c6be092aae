"""A rebuild of the quartet lists that runs out of memory (GPU test).

pfk_set_options makes the lists anew in about a dozen device allocations.
Whichever of them fails (pfk_test_fail_alloc counts down to it; the kernels
see nothing of it), the context must refuse every build, instead of running
the kernels over counts, offsets and segments of different lists, and the
same pfk_set_options called again must make the lists."""
import numpy as np
import pytest

from helpers import basis_library, pfk, random_density, water_cluster

pytestmark = pytest.mark.gpu

OLD = dict(tol_eri=1e-10, engine="os", precision="fp64")
NEW = dict(tol_eri=1e-7, engine="os", precision="mixed", fp32_bound=1e-5)


def test_failed_rebuild_is_refused_and_repeated():
    P = pfk()
    _, shells = P.shells_for(water_cluster(2, seed=5), "6-31g**", basis_library())
    eng, fresh = P.FockEngine(shells), P.FockEngine(shells)
    D = random_density(eng.nbasis, seed=7)
    old = fresh.fock_rhf(D)
    fresh.set_options(**NEW)
    new = fresh.fock_rhf(D)
    fresh.close()
    assert not np.array_equal(old, new)
    fail = eng.lib.pfk_test_fail_alloc
    fail.restype, fail.argtypes = P.ctypes.c_longlong, [P.ctypes.c_longlong]
    nth = 0
    while True:
        nth += 1
        assert nth < 200
        assert np.array_equal(eng.fock_rhf(D), old)     # also captures a graph over the old lists
        fail(nth)
        try:
            eng.set_options(**NEW)
        except P.PfkError as e:
            assert e.status in (P.PFK_ERR_CUDA, P.PFK_ERR_NOMEM)
        else:
            assert fail(0) > 0                           # fewer allocations than nth: none failed
            break
        for call in (lambda: eng.fock_rhf(D), lambda: eng.fock_uhf(D, D), lambda: eng.jk(D), eng.eri_tensor,
                     eng.quartet_count, eng.class_stats, eng.precision_stats, eng.autotune,
                     lambda: eng.rmp2_energy(np.eye(eng.nbasis), np.arange(eng.nbasis) - 4.5, 5)):
            with pytest.raises(P.PfkError) as e:
                call()
            assert e.value.status == P.PFK_ERR_STATE
        eng.set_options(**NEW)
        assert np.array_equal(eng.fock_rhf(D), new)
        eng.set_options(**OLD)
    assert nth > 10                                      # every allocation of a rebuild had its turn
    assert np.array_equal(eng.fock_rhf(D), new)
    eng.close()
