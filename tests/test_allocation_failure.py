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


def test_a_window_takes_its_memory_in_the_forward():
    """The backward sweep of a moist window allocates nothing; a forward that
    cannot have the memory fails, and the next call is not blamed for it."""
    fakecuda.run("""
_, m = make_model(3, 1, "jet_moist")
g = abi.GpuModel(m, abi.FP64)
final, bar, grad = (m.state_old.clone() for _ in range(3))
g.window_forward(m.state_old, final, 100.0, 2)
n = fake.fake_mallocs()
g.window_backward(bar, grad)
assert fake.fake_mallocs() == n, fake.fake_mallocs() - n
g.close()

for back in range(1, 4):        # the last allocations of the window's memory
    g = abi.GpuModel(m, abi.FP64)
    g.linear_combine_two_states(m.state_old, m.state_old, m.state_new, 1.0, 0.0)
    if back == 1:
        n = fake.fake_mallocs()
        g.window_forward(m.state_old, final, 100.0, 2)
        need = fake.fake_mallocs() - n
    else:
        fake.fake_fail_malloc(need - back, 0)
        try:
            g.window_forward(m.state_old, final, 100.0, 2)
            assert False, back
        except abi.GpuError as e:
            assert "allocation" in str(e), e
        fake.fake_fail_malloc(-1, 0)
        g.linear_combine_two_states(m.state_old, m.state_old, m.state_new, 1.0, 0.0)
    g.close()
""")


def test_a_failed_operator_adjoint_is_reported_once():
    fakecuda.run("""
_, m = make_model(3, 1, "jet_moist")
g = abi.GpuModel(m, abi.FP64)
args = [m.state_old, m.state_new, m.state_tendency, m.diagnostics, m.irrev]
bars = [s.clone() for s in args]
call = lambda: lib.three_band_solver_gen_densities_adj(m.state_old.ptr, m.state_new.ptr, m.state_tendency.ptr,
    m.diagnostics.ptr, m.irrev.ptr, m.config.ptr, 100.0, 0, m.grid.ptr, *[b.ptr for b in bars])
assert call() == 0, error()
g.close()
g = abi.GpuModel(m, abi.FP64)
n = fake.fake_mallocs()
assert call() == 0, error()
n = fake.fake_mallocs() - n
g.close()
g = abi.GpuModel(m, abi.FP64)
fake.fake_fail_malloc(n - 1, 0)
assert call() != 0
assert "tracer adjoint" in error(), error()
fake.fake_fail_malloc(-1, 0)
g.linear_combine_two_states(m.state_old, m.state_old, m.state_new, 1.0, 0.0)
assert call() == 0, error()
""")


def test_new_buffers_are_cleared_on_the_stream_that_uses_them():
    """The library's streams do not wait for the default stream: a clear there
    could wipe what a kernel or an upload has written meanwhile."""
    fakecuda.run("""
_, m = make_model(3, 1, "jet_moist")
g = abi.GpuModel(m, abi.FP64)
g.linear_combine_two_states(m.state_old, m.state_old, m.state_new, 1.0, 0.0)
g.manage_rkhevi(100.0, 0.0)
final, bar, grad = (m.state_old.clone() for _ in range(3))
g.window_forward(m.state_old, final, 100.0, 2)
g.window_backward(bar, grad)
m.config["momentum_diff_h"] = 1
g.manage_rkhevi(100.0, 0.0)
assert fake.fake_unordered_clears() == 0, fake.fake_unordered_clears()
""")


def test_a_mixed_run_holds_nothing_of_the_fp64_path():
    """the FP64 path's tables come with the first operator that reads them, its
    work arrays with the first FP64 step, once; without memory for them that
    call fails and the mixed step goes on"""
    fakecuda.run("""
for mountain in (False, True):
    _, m = make_model(3, 1, "jet_moist", mountain=mountain)
    lay = m.layout
    g = abi.GpuModel(m, abi.MIXED, resident=True)
    for s in (m.state_old, m.state_new, m.state_tendency):
        g.sync_to_device(s)
    bytes_ = fake.fake_live_bytes
    n, start = fake.fake_mallocs(), bytes_()
    for _ in range(2):
        g.manage_rkhevi(100.0, 0.0)
    assert fake.fake_mallocs() - n <= 1 and bytes_() == start, (fake.fake_mallocs() - n, bytes_() - start)
    lib.game_gpu_set_precision(abi.FP64)
    fake.fake_fail_malloc(3, 0)
    try:
        g.manage_rkhevi(100.0, 0.0)
        assert False
    except abi.GpuError as e:
        assert "FP64 path" in str(e), e
    fake.fake_fail_malloc(-1, 0)
    lib.game_gpu_set_precision(abi.MIXED)
    g.manage_rkhevi(100.0, 0.0)
    lib.game_gpu_set_precision(abi.FP64)
    g.manage_rkhevi(100.0, 0.0)
    per_box = (bytes_() - start) / 8 / (lay.nl * lay.nc)
    assert (46 if mountain else 37) < per_box < (50 if mountain else 40), per_box
    n = fake.fake_mallocs()
    g.manage_rkhevi(100.0, 0.0)
    lib.game_gpu_set_precision(abi.MIXED)
    g.manage_rkhevi(100.0, 0.0)
    assert fake.fake_mallocs() == n
    g.close()
""")


def test_new_lagged_fields_are_imported_without_allocating():
    """a program that hands the step another Irreversible_quantities: the import
    takes its scratch from the context (an allocation and its release cost
    0.15 ms on the smallest grid when they map and unmap memory)"""
    fakecuda.run("""
_, m = make_model(3, 1, "jet_moist")
g = abi.GpuModel(m, abi.MIXED)
g.linear_combine_two_states(m.state_old, m.state_old, m.state_new, 1.0, 0.0)
g.manage_rkhevi(100.0, 0.0)
n = fake.fake_mallocs()
m.irrev = m.irrev.clone()
g.manage_rkhevi(100.0, 0.0)
assert fake.fake_mallocs() == n, fake.fake_mallocs() - n
""")
