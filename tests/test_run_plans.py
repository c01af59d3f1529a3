"""Which plans of folded inference runs are kept (host rule)."""
import threading


def _net():
    from deeplearning4j_b200.nn.graph import ComputationGraph
    return ComputationGraph.__new__(ComputationGraph)


def test_recently_used_shapes_stay_and_starts_do_not_count():
    net, made = _net(), []

    def plan(shape, start):
        return net._run_plan(shape, start, lambda: made.append((shape, start)) or {"n": 0})
    for start in range(20):                       # many starts of one shape, none with a run
        plan("a", start)
    n = len(made)
    for start in range(20):
        plan("a", start)
    assert len(made) == n
    for s in "bcdefgh":
        plan(s, 0)
    plan("a", 0)                                  # a hit keeps it
    plan("i", 0)                                  # the ninth shape: "b" goes
    n = len(made)
    plan("a", 0)
    assert len(made) == n and len(net._run_plans) == 8
    plan("b", 0)
    assert len(made) == n + 1


def test_threads_share_a_network():
    net, errors = _net(), []

    def work(k):
        try:
            for i in range(3000):
                p = net._run_plan((i * 7 + k) % 23, i % 5, lambda: {"n": (i * 7 + k) % 23})
                assert p["n"] == (i * 7 + k) % 23
        except Exception as e:                    # noqa: BLE001
            errors.append(e)
    ts = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    [t.start() for t in ts], [t.join() for t in ts]
    assert not errors
