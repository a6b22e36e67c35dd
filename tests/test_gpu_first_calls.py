"""First calls of a process from several threads and streams at once: each kernel is set up by whichever comes first."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import threading, torch
import l_inf_dist_net_v2_b200 as ldn
torch.manual_seed(0)
x, w = torch.rand(512, 2048, 1, device="cuda"), torch.randn(2560, 2048, device="cuda")
g = torch.randn(512, 2560, 1, device="cuda")
image, filters = torch.rand(8, 300, 81, device="cuda"), torch.randn(64, 300, device="cuda")
torch.cuda.synchronize()
results, barrier = {}, threading.Barrier(6)

def work(k):
    with torch.cuda.stream(torch.cuda.Stream()):
        a, b = x.clone().requires_grad_(), w.clone().requires_grad_()
        barrier.wait()
        out = []
        for p in (8.0, 4.0, 37.5):
            y = ldn.norm_dist(a, b, p)
            out += [y.detach(), *torch.autograd.grad(y, (a, b), g)]
        # (values only: gradients at p = inf are added up in no fixed order)
        out += [ldn.norm_dist(x, w, float("inf")), ldn.norm_dist(image, filters, float("inf"))]
        torch.cuda.current_stream().synchronize()
        results[k] = out

threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
[t.start() for t in threads]
[t.join() for t in threads]
assert len(results) == 6
for k in range(1, 6):
    for i, (a, b) in enumerate(zip(results[0], results[k])):
        assert torch.equal(a, b), (k, i)
print("same")
"""


def test_threads():
    r = subprocess.run([sys.executable, "-c", PROGRAM], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("same"), r.stderr[-2000:]
