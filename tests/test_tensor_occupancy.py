"""One CTA of the tensor step per SM, whatever the compiler makes of its registers: each
holds all of the SM's tensor memory, and launches of many generations wait for each
other's CTAs.  Read from the source, since it takes no GPU to say."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def source(name):
    return open(os.path.join(ROOT, "cat_cpu_b200", "csrc", name)).read()


def test_shared_memory_keeps_ctas_apart():
    kb = int(re.search(r"constexpr int kSmemFloor = (\d+) \* 1024;", source("k_tensor.cu")).group(1))
    # 228 KB per SM, 1 KB of it reserved per CTA, 227 KB at most for one
    assert 2 * (kb + 1) > 228 and kb <= 227


def test_next_launch_starts_after_the_allocation():
    s = source("tensor_step.cuh")
    kernel = s[s.index("k_tensor_step(const __grid_constant__"):]
    alloc, barrier, chain = (kernel.index(x) for x in ("tmem_alloc(tmem_slot", "__syncthreads();", "chain_wait();"))
    assert alloc < barrier < chain
    assert kernel.count("chain_wait();") == 1 and "launch_dependents" not in s
