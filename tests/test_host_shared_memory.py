"""Kernels with more than 48 KB of dynamic shared memory need their limit raised on
the device that runs them."""
import fake_device


def test_networks_on_two_devices(tmp_path):
    fake_device.run("""
        rng = np.random.default_rng(3)
        # (inputs, bins): the staged kernels, and the general ones beyond 48 KB
        for kind, P, B in (("additive", 16, 72), ("affine", 264, 6152)):
            for device in (0, 1):
                s = Surrogate(P, B, hidden=(24, 40), batch_max=64, device=device)
                th = rng.normal(size=(300, P))
                logs = 0.1 * rng.normal(size=(300, B))
                s.fit_additive(th, logs, log_ratio=logs) if kind == "additive" else s.fit_affine(th, logs)
                s.attach(np.ones(B), None if kind == "additive" else np.ones(B), N.GW_LLH_POISSON)
                s.set_chain(np.eye(P))
                s.value_grad(th[:8])
                s.stat_llh(th[:8])
                s.reserve(64)
                s.append(th[:32], np.exp(logs[:32]))
                s.train(epochs=1, lr=1e-3, batch=32)
                s.close()
                lines = log()
                assert any(f"device {device}" in x for x in lines)
                assert not [x for x in lines if x.startswith("refused")], (kind, device)
    """, tmp_path)


def test_a_refused_limit_is_reported(tmp_path):
    fake_device.run("""
        _fake.fake_set_optin(64 * 1024)
        m = MLP([16, 24, 72], batch_max=64)
        m.init(1)
        try:
            m.forward(np.zeros((8, 16), np.float32))
        except N.GwError as e:
            assert "invalid argument" in str(e), e
        else:
            raise AssertionError("no error")
        assert not [x for x in log() if x.startswith("refused")]  # nothing was launched with it
    """, tmp_path)


def test_engines_of_different_sizes_side_by_side(tmp_path):
    fake_device.run("""
        wl = Workload("mixed", seed=3)
        def small_last(build, use):
            for order in ((0, 1), (1, 0)):
                engines = [build(i) for i in order]
                log()
                for e in engines:
                    use(e)
                assert not [x for x in log() if x.startswith("refused")], order
                for e in engines:
                    e.close()
        for precision in ("fp32", "fp64", "df64"):
            # tiles of two sizes, through the one-point and the batched kernels
            for k in (1, 4, 64):
                small_last(lambda i: Engine.from_workload(wl, precision=precision, k_max=k, tile_bytes=(0, 8192)[i]),
                           lambda e: e.eval(wl.draw_points(k, 1)))
            # numbers of parameters
            def engine(i):
                e = Engine(4, (8192, 16)[i], 4, precision=precision)
                e.set_event_indices(np.arange(4, dtype=np.int32))
                e.initialize()
                return e
            small_last(engine, lambda e: e.eval(np.zeros((1, e.n_params))))
    """, tmp_path)
