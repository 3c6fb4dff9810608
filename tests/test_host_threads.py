"""The library's helper threads (planning on several cores), on the CPU: a process forked from one that has
helpers plans on its own, with the same results."""
import os
import subprocess
import sys
import textwrap

import pytest

FORK = textwrap.dedent("""
    import os, signal, threading
    from fgkl_b200 import synthetic
    from fgkl_b200.shard import region_costs

    few, many = (synthetic.workload(2, seed=s, regions=n, threads=1) for s, n in ((4, 3), (5, 64)))
    expected = region_costs(many).tolist()  # leaves idle helpers behind
    stop = threading.Event()
    busy = None
    if {busy}:  # helpers at work, and their lock taken now and then, while the process forks
        busy = threading.Thread(target=lambda: [region_costs(few) for _ in iter(stop.is_set, True)])
        busy.start()
    for _ in range(4):
        region_costs(few)
        child = os.fork()
        if child == 0:
            signal.alarm(30)
            same = all(region_costs(many).tolist() == expected for _ in range(10))
            os._exit(0 if same else 1)
        status = os.waitpid(child, 0)[1]
        assert status == 0, status
    stop.set()
    if busy:
        busy.join()
    assert region_costs(many).tolist() == expected
""")


@pytest.mark.parametrize("busy", [False, True])
def test_a_forked_process_plans_with_helpers_of_its_own(busy):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    run = subprocess.run([sys.executable, "-W", "ignore::DeprecationWarning", "-c", FORK.format(busy=busy)], cwd=root, timeout=300,
                         capture_output=True, text=True)
    assert run.returncode == 0, run.stderr
