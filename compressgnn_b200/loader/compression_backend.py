"""Backend choice for the grammar compressor (mirror of the reference's
``loader/compression_backend.py:6-40``).  Two compressors produce the same arrays: the host one in
``libcgnn_host.so`` (``'cpu'``) and the device one in ``libcgnn_b200.so`` (``'cuda'``,
``cgnn_compress_csr_batch``).  ``'auto'`` takes the device when one is usable, as the reference does
when its CUDA extension is installed."""
import operator

import numpy as np

from .. import offline


def _cuda_usable():
    try:
        import torch
        from .._lib import lib
        if not torch.cuda.is_available():
            return False
        lib()
        return True
    except (ImportError, OSError):
        return False


def resolve_backend(backend):
    if backend not in ('auto', 'cpu', 'cuda'):
        raise ValueError("compression_backend must be 'auto', 'cpu', or 'cuda'")
    if backend == 'cpu':
        return 'cpu'
    if _cuda_usable():
        return 'cuda'
    if backend == 'cuda':
        raise RuntimeError('CUDA compression requested but no usable CUDA device (or libcgnn_b200.so) is available')
    return 'cpu'


# A copy between pageable host memory and the device goes through the driver's own stage at about 11 GB/s, one host
# thread moving the bytes (27 MB of edges: 2.6 ms).  In parts through two page-locked stages the host side of a part is
# done by torch's threads while the part before it is on the link.  The stages are torch's, which
# keeps page-locked memory of this size for the next caller; up to one part the plain copy is as fast, and where there
# is no page-locked memory to be had it takes all.
STAGE_BYTES = 4 << 20


def _parts(tensor):
    step = STAGE_BYTES // tensor.element_size()
    return [slice(at, at + step) for at in range(0, tensor.numel(), step)]


def _stages(tensor):
    """Two page-locked stages, or None for the plain copy."""
    import torch
    if tensor.nbytes <= STAGE_BYTES:
        return None
    step = STAGE_BYTES // tensor.element_size()
    try:
        return [(torch.empty(step, dtype=tensor.dtype, device="cpu", pin_memory=True), torch.cuda.Event()) for _ in range(2)]
    except RuntimeError:
        return None


def _to_device(host):
    """One-dimensional host tensor on the current device."""
    import torch
    stages = _stages(host)
    if stages is None:
        return host.cuda()
    out = torch.empty_like(host, device="cuda")
    for i, part in enumerate(_parts(host)):
        stage, sent = stages[i % 2]
        sent.synchronize()  # (an event not recorded yet is complete)
        stage = stage[:host[part].numel()]
        stage.copy_(host[part])
        out[part].copy_(stage, non_blocking=True)
        sent.record()
    return out


def _to_host(device):
    """One-dimensional device tensor in pageable host memory, complete on return."""
    import torch
    stages = _stages(device)
    if stages is None:
        return device.cpu()
    out, parts = torch.empty(device.shape, dtype=device.dtype, device="cpu"), _parts(device)
    for i in range(len(parts) + 1):
        if i < len(parts):
            stage, arrived = stages[i % 2]
            stage[:device[parts[i]].numel()].copy_(device[parts[i]], non_blocking=True)
            arrived.record()
        if i > 0:
            stage, arrived = stages[(i - 1) % 2]
            arrived.synchronize()
            out[parts[i - 1]].copy_(stage[:out[parts[i - 1]].numel()])
    return out


def _compress_on_device(vlist, elist, rounds, frequency):
    import torch
    from .. import runtime
    vlist, elist = offline._i64(vlist), offline._i64(elist)
    def require_int32_range():
        if vlist.size < 1 or (elist.size and (elist.max() > np.iinfo(np.int32).max or elist.min() < 0)):
            raise ValueError("CSR value exceeds int32 range")

    # The compressor looks at every edge of the rows and refuses a value outside the graph; two more passes over
    # the host array (2.3 ms at 3.4 M edges) are needed only to name the error, or for edges behind the last row.
    if vlist.size < 1 or vlist[-1] != elist.size:
        require_int32_range()
    if vlist.size > 1 and vlist[-1] > elist.size:
        raise RuntimeError(runtime._BAD_ROW_POINTERS)
    # Runtime failures (out of memory included) propagate; nothing falls back to the host.
    try:
        v, e, n, r = runtime._compress_rows(_to_device(torch.from_numpy(vlist)), _to_device(torch.from_numpy(elist)), rounds,
                                            frequency)
    except RuntimeError:
        require_int32_range()
        raise
    return _to_host(v).numpy(), _to_host(e).numpy(), n, r


def compress_graph_csr(vlist, elist, min_pair_frequency=16, backend='auto', threads=4, rounds=12):
    frequency = operator.index(min_pair_frequency)
    threads = operator.index(threads)
    rounds = operator.index(rounds)
    if threads < 1 or rounds < 1:
        raise ValueError('compression_threads and compression_rounds must be positive')
    selected = resolve_backend(backend)
    if frequency < 3:
        raise ValueError('Batch compression needs min_pair_frequency >= 3')
    if selected == 'cuda':
        return _compress_on_device(vlist, elist, rounds, frequency)
    return offline.compress_csr_batch(vlist, elist, threads=threads, rounds=rounds,
                                      min_pair_frequency=frequency)
