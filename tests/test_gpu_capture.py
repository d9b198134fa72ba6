"""Stream capture after one warm-up call of another size, and in a process that has made no call at all: no size may allocate or synchronise on
its first launch.  Processes of their own, since a kernel's first launch happens once; what a process captures first is what differs."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import sys, torch, kiln_b200
dev = torch.device("cuda")
gen = torch.Generator(device=dev)
gen.manual_seed(3)

def prepare(kind, m):
    k, n = (2560, 512) if kind == "narrow" else (2560, 4096)
    g = -1 if kind == "per_column" else 128
    words = torch.randint(-2 ** 31, 2 ** 31 - 1, (k // 16, 2 * n), dtype=torch.int32, device=dev, generator=gen)
    scales = (0.01 * torch.rand((1 if g == -1 else k // 128, n), device=dev, generator=gen) + 1e-3).to(torch.float16)
    proj = kiln_b200.MarlinPackedProj(words, scales, g, k, n)
    x = torch.randn((m, k), device=dev, generator=gen).to(torch.bfloat16)
    la, lb = torch.randn((16, k), device=dev, generator=gen).to(torch.bfloat16), torch.randn((n, 16), device=dev, generator=gen).to(torch.bfloat16)
    return {"lora": lambda: kiln_b200.matmul_bf16_lora(x, proj, la, lb, 0.5), "swiglu": lambda: kiln_b200.swiglu_gate_up(x, proj),
            "grouped": lambda: kiln_b200.grouped_matmul_bf16([x, x], [proj, proj])[1]}.get(kind, lambda: kiln_b200.matmul_bf16(x, proj))

calls = [prepare(*case.split(":")[:1], int(case.split(":")[1])) for case in sys.argv[2:]]
if sys.argv[1] == "warm":
    prepare("plain", 1)()
torch.cuda.synchronize()
for case, call in zip(sys.argv[2:], calls):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, call()), case
print("captured")
"""
CASES = ["plain:9", "lora:5", "plain:512", "narrow:64", "lora:40", "swiglu:16", "swiglu:300", "per_column:100", "grouped:16", "plain:64", "plain:2048"]


@pytest.mark.parametrize("before,first", [("warm", 0), ("warm", 1), ("warm", 2), ("cold", 0)])
def test_any_size_is_captured(cuda_device, before, first):
    done = subprocess.run([sys.executable, "-c", CHILD, before, *CASES[first:], *CASES[:first]], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0 and "captured" in done.stdout, done.stderr[-2000:]
