"""Set-up work (clears, uploads) and the kernels that read it: in one stream, or
apart by a synchronisation.  The network's and the engine's streams do not wait
for the legacy default stream, where cudaMemset returns before it is done and the
last part of a copy from pageable memory may still be in flight."""
import fake_device


def test_network_setup_is_ordered_before_its_kernels(tmp_path):
    fake_device.run("""
        rng = np.random.default_rng(3)
        P, B, K = 16, 72, 13
        for kind in ("additive", "affine"):
            s = Surrogate(P, B, hidden=(24, 40), batch_max=64)
            th = rng.normal(size=(200, P))
            logs = 2.0 + 0.1 * rng.normal(size=(200, B))
            s.fit_additive(th, logs, log_ratio=0.1 * rng.normal(size=(200, B))) if kind == "additive" else s.fit_affine(th, logs)
            s.attach(np.ones(B), None if kind == "additive" else np.ones(B), N.GW_LLH_POISSON)
            s.set_chain(np.eye(P), np.zeros(P), np.eye(P))
            s.value_grad(th[:K])  # its buffers are made by the first call
            s.stat_llh(th[:K])
            s.substeps(th[:K], None, 2, 5)
            s.reserve(128)
            s.append(th[:64], np.exp(logs[:64]))
            s.train(epochs=2, lr=1e-3, batch=32)
            w, b = s.mlp.get_layer(0)
            s.mlp.set_layer(0, w, b)
            s.mlp.forward(th[:16].astype(np.float32))
            s.mlp.gradients(th[:16].astype(np.float32), logs[:16].astype(np.float32))
            s.close()
        lines = log()
        assert any("launch" in x for x in lines)
        bad = sorted({x for x in lines if x.startswith("unordered")})
        assert not bad, bad
    """, tmp_path)


def test_engine_setup_is_ordered_before_its_kernels(tmp_path):
    fake_device.run("""
        wl = Workload("mixed", seed=3)
        for precision in ("fp32", "fp64", "df64"):
            e = Engine.from_workload(wl, precision=precision, k_max=8)
            e.eval(wl.draw_points(1, 1))
            e.set_data(wl.data)
            e.eval(wl.draw_points(8, 1))
            e.autotune(1)
            e.autotune(8)
            e.eval(wl.draw_points(8, 1))
            e.set_event_weight_copy(True)
            e.eval(wl.draw_points(1, 1))
            e.event_weights()
            e.close()
        lines = log()
        assert any("launch" in x for x in lines)
        bad = sorted({x for x in lines if x.startswith("unordered")})
        assert not bad, bad
    """, tmp_path)
