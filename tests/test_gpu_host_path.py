"""The native host path of the Python entry points at its edges: calls that it must leave to the Python path, or must not change."""
import subprocess
import sys

import pytest
import torch

import kiln_b200

pytestmark = pytest.mark.gpu


def _child(code):
    """Runs code in a process of its own (what it tests would end the process) and returns its output."""
    done = subprocess.run([sys.executable, "-c", "import torch, kiln_b200\ndev = torch.device('cuda')\n" + code], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, f"exit code {done.returncode}\n{done.stderr[-2000:]}"
    return done.stdout


def test_a_problem_without_rows_of_weights_is_refused(cuda_device):
    out = _child("""
try:
    kiln_b200.marlin_w4a16_gemm(torch.empty((4, 0), dtype=torch.bfloat16, device=dev), torch.empty((0, 512), dtype=torch.int32, device=dev),
                                torch.empty((0, 256), dtype=torch.float16, device=dev), 128)
except kiln_b200.KilnMarlinError as e:
    print(e)
""")
    assert "k=0 must be divisible by groupsize=128" in out


class _Offloaded:
    """A projection whose tensors are brought to the GPU whenever they are read."""

    def __init__(self, proj):
        self.b_cpu, self.s_cpu, self.groupsize, self.k, self.n = proj.b_packed.cpu(), proj.scales.cpu(), proj.groupsize, proj.k, proj.n

    @property
    def b_packed(self):
        return self.b_cpu.to("cuda")

    @property
    def scales(self):
        return self.s_cpu.to("cuda")


def test_weights_made_on_each_read_live_until_the_launch(cuda_device):
    """Memory of a weight that nobody holds goes to the next tensor of its size: the second projection of a group, the output, the
    workspace.  Sizes on both sides of the allocator's 1 MB, so that each of those can happen."""
    gen = torch.Generator().manual_seed(5)
    for k, n, m in [(512, 256, 64), (512, 256, 5), (2560, 2560, 64), (1024, 2048, 1024)]:
        def proj():
            b = torch.randint(-2 ** 31, 2 ** 31 - 1, (k // 16, 2 * n), dtype=torch.int32, generator=gen)
            s = (0.01 * torch.rand((k // 128, n), generator=gen) + 1e-3).to(torch.float16)
            return kiln_b200.MarlinPackedProj(b.to(cuda_device), s.to(cuda_device), 128, k, n)

        p, q = proj(), proj()
        x = torch.randn((m, k), generator=gen).to(torch.bfloat16).to(cuda_device)
        la, lb = torch.randn((16, k), generator=gen).to(torch.bfloat16).to(cuda_device), torch.randn((n, 16), generator=gen).to(torch.bfloat16).to(cuda_device)

        def calls(p, q, x=x):
            return [kiln_b200.matmul_bf16(x, p), kiln_b200.swiglu_gate_up(x, p), kiln_b200.matmul_bf16_lora(x, p, la, lb, 0.5),
                    *kiln_b200.grouped_matmul_bf16([x, x], [p, q])]

        want = calls(p, q)
        for _ in range(5):
            for got, ref in zip(calls(_Offloaded(p), _Offloaded(q)), want):
                assert torch.equal(got, ref)
            for got, ref in zip(calls(_Offloaded(p), _Offloaded(q), x.t().contiguous().t()), want):  # the Python path, which copies x
                assert torch.equal(got, ref)


def test_an_error_while_the_gil_is_free_arrives_as_a_python_exception(cuda_device):
    """pack_from_gptq reads a counter back, which is refused while the stream is being captured."""
    out = _child("""
q = torch.zeros((16, 256), dtype=torch.int32, device=dev)
z = torch.full((1, 32), -0x77777778, dtype=torch.int32, device=dev)
s = torch.ones((1, 256), dtype=torch.float16, device=dev)
assert kiln_b200.pack_from_gptq(q, z, s) is not None
try:
    with torch.cuda.graph(torch.cuda.CUDAGraph()):
        try:
            kiln_b200.pack_from_gptq(q, z, s)
        except RuntimeError:
            print("raised", flush=True)
            raise
except RuntimeError:
    print("alive", flush=True)
""")
    assert out.split() == ["raised", "alive"]


def test_out_of_memory_keeps_its_type(cuda_device):
    """What a server catches to evict and try again: for an output, a workspace and a packed weight alike."""
    out = _child("""
torch.cuda.set_per_process_memory_fraction((64 << 20) / torch.cuda.mem_get_info()[1])
proj = kiln_b200.pack_from_bf16(torch.zeros((128, 1024), dtype=torch.bfloat16, device=dev))
x = torch.zeros((8192, 128), dtype=torch.bfloat16, device=dev)
w = torch.zeros((4096, 4096), dtype=torch.bfloat16, device=dev)
big = kiln_b200.MarlinPackedProj(proj.b_packed.repeat(1, 8), proj.scales.repeat(1, 8), 128, 128, 8192)
for call in (lambda: kiln_b200.matmul_bf16(x, big), lambda: kiln_b200.swiglu_gate_up(x, big), lambda: kiln_b200.grouped_matmul_bf16([x], [big]),
             lambda: [kiln_b200.pack_from_bf16(w) for _ in range(8)]):
    try:
        held = call()
        print("allocated")
    except torch.OutOfMemoryError as e:
        print("C++" if "Exception raised from" in str(e) else "out of memory")
    held = None
""")
    assert out.split("\n")[:4] == ["out of memory"] * 4


def test_a_group_size_beyond_a_long_is_refused(cuda_device):
    w = torch.randn((128, 256), device=cuda_device).to(torch.bfloat16)
    proj = kiln_b200.pack_from_bf16(w, -1)
    x = torch.zeros((3, 128), dtype=torch.bfloat16, device=cuda_device)
    for g in (2 ** 70, -2 ** 63 - 1, 2 ** 32 + 128):
        for call in (lambda: kiln_b200.marlin_w4a16_gemm(x, proj.b_packed, proj.scales, g), lambda: kiln_b200.pack_from_bf16(w, g),
                     lambda: kiln_b200.matmul_bf16(x, kiln_b200.MarlinPackedProj(proj.b_packed, proj.scales, g, 128, 256))):
            with pytest.raises(kiln_b200.KilnMarlinError, match="groupsize must be -1 or 128"):
                call()
        qzeros = torch.full((1, 32), -0x77777778, dtype=torch.int32, device=cuda_device)
        assert kiln_b200.pack_from_gptq(torch.zeros((16, 256), dtype=torch.int32, device=cuda_device), qzeros, proj.scales, g) is None


def test_gptq_tensors_that_have_to_be_copied_do_not_overlap(cuda_device):
    """Neither tensor is contiguous: both copies have to live until the repack is enqueued."""
    gen = torch.Generator(device=cuda_device)
    gen.manual_seed(1)
    for k, n in [(1024, 1024), (256, 256), (4096, 2048)]:
        qw = torch.randint(-2 ** 31, 2 ** 31 - 1, (k // 8, n), dtype=torch.int32, device=cuda_device, generator=gen)
        qz = torch.full((k // 128, n // 8), -0x77777778, dtype=torch.int32, device=cuda_device)
        s = torch.rand((k // 128, n), device=cuda_device, generator=gen).to(torch.float16)
        want = kiln_b200.pack_from_gptq(qw, qz, s)
        got = kiln_b200.pack_from_gptq(qw.t().contiguous().t(), qz.t().contiguous().t(), s.t().contiguous().t())
        assert torch.equal(got.b_packed, want.b_packed) and torch.equal(got.scales, want.scales)
