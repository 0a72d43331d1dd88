"""Which kernels a call launches, for tests of a dispatch."""
import torch


def kernel_counts(f, tries=4):
    """{name: launches} of f()'s device activities, by the profiler; f again if
    it has seen no kernel at all."""
    torch.zeros(1, device="cuda")
    for _ in range(tries):
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
            f()
            torch.cuda.synchronize()
        counts = {e.key: e.count for e in p.key_averages()}
        if any("k_" in k for k in counts):
            return counts
    raise AssertionError("the profiler saw no kernel: %s" % sorted(counts))


def launched(counts, name):
    """Launches of the kernels whose name holds `name`."""
    return sum(n for k, n in counts.items() if name in k)
