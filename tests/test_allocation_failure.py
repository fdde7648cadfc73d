"""A device allocation that fails in game_gpu_init: an error, no kernel on the
pointers that are missing, everything given back, and the next init works.
Without a GPU (fakecuda.py)."""
import fakecuda


def test_init_reports_a_failed_allocation_and_launches_nothing():
    fakecuda.run("""
_, m = make_model(3, 1, "jet_moist", mountain=True)
init = lambda: lib.game_gpu_init(3, 26, 1, m.grid.ptr, m.dualgrid.ptr)
assert init() == 0, error()
total = fake.fake_mallocs()
assert lib.game_gpu_finalize() == 0 and fake.fake_live_bytes() == 0
assert total > 100
for k in [0, 1, total // 3, total // 2] + list(range(total - 24, total)):
    launched = fake.fake_launches()
    fake.fake_fail_malloc(k, 0)
    assert init() != 0, k
    assert "allocation" in error(), (k, error())
    assert fake.fake_launches() == launched, k
    assert fake.fake_live_bytes() == 0, k
    fake.fake_fail_malloc(-1, 0)
assert init() == 0, error()
""")
