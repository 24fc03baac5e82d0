"""On-disk forms written by the reference, loaded and run on the GPU. Needs a B200.

tests/golden/sidecar_small.tq1g128 and .lut23 were written by the reference's own writers
(src/bonsai_tq1/format.py:149-246, src/bonsai_tq1/lut23_reorder.py:42-123,323-334; see make_golden.py).
Each tensor goes reader -> PackedLinear.load_blocks (device scan) -> tq1_matmul and is compared with the
oracle, at batch 1 and 5.
"""

import numpy as np
import pytest
import torch

from oracle import tq1_oracle as o
from ternel_b200 import loaders
from tests.conftest import GOLDEN
from tests.gpu_util import random_blocks

pytestmark = pytest.mark.gpu

NAMES = ("blk.0.ffn_down.weight", "blk.0.ssm_a.weight")


def _run(blocks, name):
    from ternel_b200.layout import PackedTensorLayout
    from ternel_b200.modules import PackedLinear
    rows, columns = blocks.shape[0], blocks.shape[1] * 128
    layer = PackedLinear(PackedTensorLayout.for_tensor(rows, columns), device="cuda", out_dtype=torch.float32)
    layer.load_blocks(blocks)                      # runs the fail-closed byte scan on the device
    rng = np.random.default_rng(len(name))
    for batch in (1, 5):
        x = rng.standard_normal((batch, columns)).astype(np.float16)
        got = layer(torch.from_numpy(x).cuda()).cpu().numpy()
        want = o.float64_matmul(blocks, x, rows=rows, columns=columns)
        assert got.shape == (batch, rows)
        assert o.normalised_error(got, want) < 1e-5, (name, batch)


def test_sidecar_tensors_run_on_the_gpu():
    _, manifest = loaders.read_sidecar(GOLDEN / "sidecar_small.tq1g128")
    for name in NAMES:
        _run(loaders.load_sidecar_tensor(GOLDEN / "sidecar_small.tq1g128", manifest, name), name)


def test_lut23_sidecar_tensors_run_on_the_gpu():
    _, manifest = loaders.read_lut23_sidecar(GOLDEN / "sidecar_small.lut23")
    for name in NAMES:
        _run(loaders.load_lut23_tensor(GOLDEN / "sidecar_small.lut23", manifest, name), name)


@pytest.mark.parametrize("rows,columns", [(1, 128), (48, 5120), (100, 640), (256, 128), (768, 1408)])
def test_tiled_pair_is_converted_on_the_gpu(rows, columns):
    """One tile or several, rows that fill no thread block: the same blocks as the host converter's; an illegal byte
    in any slot is counted and leaves the module as it was."""
    from ternel_b200.format import FormatError
    from ternel_b200.layout import PackedTensorLayout, pack_blocks
    from ternel_b200.modules import PackedLinear
    layout = PackedTensorLayout.for_tensor(rows, columns)
    blocks, _ = random_blocks(rows, columns, seed=rows)
    codes, scales = pack_blocks(blocks, layout=layout)
    module = PackedLinear(layout, device="cuda")
    module.load_tiled(codes, scales)
    assert np.array_equal(module.blocks.cpu().numpy(), blocks)
    module.load_tiled(torch.from_numpy(codes), torch.from_numpy(scales.view(np.int16)).cuda())
    assert np.array_equal(module.blocks.cpu().numpy(), blocks)
    codes[0, 0, 0, 0], codes[-1, -1, 24, -1], codes[-1, -1, 25, 0] = 243, 255, 27
    with pytest.raises(FormatError, match=r"regular=2 \(max 242\), tail=1 \(max 26\)"):
        module.load_tiled(codes, np.zeros_like(scales))
    assert np.array_equal(module.blocks.cpu().numpy(), blocks)


def test_loaded_blocks_are_there_on_every_stream():
    """A load returns when the blocks are written, as a copy from the host does: nothing is left in flight on the loading
    stream, so another stream or thread may use the module at once."""
    from ternel_b200.layout import PackedTensorLayout, pack_blocks
    from ternel_b200.modules import PackedLinear
    layout = PackedTensorLayout.for_tensor(17408, 5120)
    blocks, _ = random_blocks(17408, 5120, seed=1)
    codes, scales = pack_blocks(blocks, layout=layout)
    codes, scales = torch.from_numpy(codes).cuda(), torch.from_numpy(scales.view(np.int16)).cuda()
    module = PackedLinear(layout, device="cuda")
    torch.cuda.synchronize()
    for _ in range(5):
        loading, using = torch.cuda.Stream(), torch.cuda.Stream()
        with torch.cuda.stream(loading):
            module.load_tiled(codes, scales)
            assert loading.query()
        with torch.cuda.stream(using):
            seen = module.blocks.clone()
        torch.cuda.synchronize()
        assert np.array_equal(seen.cpu().numpy(), blocks)
        module.blocks.zero_()
        torch.cuda.synchronize()


def test_read_only_arrays_are_converted_on_the_gpu(monkeypatch):
    """What a file mapping or a bytes object holds takes the same way as arrays that can be written."""
    from ternel_b200 import modules
    from ternel_b200.layout import PackedTensorLayout, pack_blocks
    layout = PackedTensorLayout.for_tensor(768, 1408)
    blocks, _ = random_blocks(768, 1408, seed=4)
    codes, scales = pack_blocks(blocks, layout=layout)
    codes, scales = (np.frombuffer(a.tobytes(), dtype=a.dtype).reshape(a.shape) for a in (codes, scales))
    module = modules.PackedLinear(layout, device="cuda")
    monkeypatch.setattr(modules, "unpack_blocks", None)                 # the host converter
    module.load_tiled(codes, scales)
    assert np.array_equal(module.blocks.cpu().numpy(), blocks)


def test_blocks_off_the_word_grid_are_loaded_too():
    """A module whose blocks are a view into a flat buffer at an odd address, which the conversion on the GPU does not take."""
    from ternel_b200.layout import PackedTensorLayout, pack_blocks
    from ternel_b200.modules import PackedLinear
    layout = PackedTensorLayout.for_tensor(48, 640)
    blocks, _ = random_blocks(48, 640, seed=2)
    module = PackedLinear(layout, device="cuda")
    flat = torch.zeros(blocks.size + 4, dtype=torch.uint8, device="cuda")
    for shift in (1, 2, 3, 0):
        module.blocks = flat[shift:shift + blocks.size].view(blocks.shape)
        module.load_tiled(*pack_blocks(blocks, layout=layout))
        assert np.array_equal(module.blocks.cpu().numpy(), blocks)
        flat.zero_()


@pytest.mark.parametrize("staging_bytes", (65536, 100_000, 8 << 20))
@pytest.mark.parametrize("sizes", ((1, 0), (16384, 1), (65537, 5), (700_001, 70_000), (5_324_800, 409_600), (0, 9_000_001)))
def test_upload_through_staging_of_any_size(sizes, staging_bytes):
    """Fewer bytes than a piece, ends inside a piece, many turns of the staging, and the pieces of two arrays side by side."""
    from ternel_b200 import _native
    rng = np.random.default_rng(sum(sizes))
    hosts = [rng.integers(0, 256, size + 3, dtype=np.uint8)[3:] for size in sizes]         # off the 16-byte grid
    devices = [torch.zeros(size + 64, dtype=torch.uint8, device="cuda") for size in sizes]
    staging = torch.empty(staging_bytes, dtype=torch.uint8, pin_memory=True)
    lib, stream = _native.lib(), torch.cuda.current_stream().cuda_stream
    rc = lib.tq1_upload_pair(devices[0].data_ptr(), hosts[0].ctypes.data, sizes[0], devices[1].data_ptr(), hosts[1].ctypes.data,
                             sizes[1], staging.data_ptr(), staging.numel(), stream)
    assert rc == 0
    for host, device in zip(hosts, devices):
        got = device.cpu().numpy()
        assert np.array_equal(got[:host.size], host) and not got[host.size:].any()
    assert lib.tq1_upload_pair(devices[0].data_ptr(), hosts[0].ctypes.data, 1, None, None, 0, staging.data_ptr(), 1024, stream) != 0


def _tiled_module(rows, columns, seed):
    from ternel_b200.layout import PackedTensorLayout, pack_blocks
    from ternel_b200.modules import PackedLinear
    layout = PackedTensorLayout.for_tensor(rows, columns)
    blocks, _ = random_blocks(rows, columns, seed=seed)
    return PackedLinear(layout, device="cuda"), blocks, pack_blocks(blocks, layout=layout)


def test_load_tiled_without_pinned_memory(monkeypatch):
    """Where no staging can be pinned, the arrays are uploaded as they are."""
    module, blocks, tiled = _tiled_module(768, 1408, 5)
    empty, refused = torch.empty, []

    def no_pinned(*args, **kwargs):
        if kwargs.get("pin_memory"):
            refused.append(args)
            raise RuntimeError("out of pinned memory")
        return empty(*args, **kwargs)
    monkeypatch.setattr(torch, "empty", no_pinned)
    module.load_tiled(*tiled)
    assert refused and np.array_equal(module.blocks.cpu().numpy(), blocks)


@pytest.mark.parametrize("device", ("cuda", "meta", "cpu"))
def test_load_tiled_under_a_default_device(monkeypatch, device):
    """The staging is pinned host memory whatever tensors are made on by default."""
    module, blocks, tiled = _tiled_module(768, 1408, 7)
    empty, staged = torch.empty, []

    def noted(*args, **kwargs):
        tensor = empty(*args, **kwargs)
        if kwargs.get("pin_memory"):
            staged.append(tensor.is_pinned() and tensor.data_ptr() != 0)
        return tensor
    monkeypatch.setattr(torch, "empty", noted)
    with torch.device(device):
        module.load_tiled(*tiled)
    assert staged == [True] and np.array_equal(module.blocks.cpu().numpy(), blocks)


@pytest.mark.parametrize(("rows", "columns", "staged"), ((48, 512, 0), (192, 1280, 0), (496, 640, 1)))
def test_small_arrays_are_not_staged(monkeypatch, rows, columns, staged):
    """Below 64 KiB the driver's own way is the faster one."""
    module, blocks, tiled = _tiled_module(rows, columns, 8)
    empty, pinned = torch.empty, []
    monkeypatch.setattr(torch, "empty", lambda *a, **k: (pinned.append(a) if k.get("pin_memory") else None, empty(*a, **k))[1])
    module.load_tiled(*tiled)
    assert len(pinned) == staged and np.array_equal(module.blocks.cpu().numpy(), blocks)


@pytest.mark.parametrize("fails", (False, True))
def test_staging_is_held_until_its_transfers_are_done(monkeypatch, fails):
    """The pool of pinned memory does not know of them: the staging goes back to it after the stream has been waited for."""
    import weakref
    from ternel_b200 import _native
    module, blocks, tiled = _tiled_module(768, 1408, 6)
    empty, held, seen, synchronize = torch.empty, [], [], torch.cuda.Stream.synchronize

    def noted(*args, **kwargs):
        tensor = empty(*args, **kwargs)
        if kwargs.get("pin_memory"):
            held.append(weakref.ref(tensor))
        return tensor

    class Library:
        def __getattr__(self, name):
            return getattr(real, name)

        def tq1_load_tiled_device(self, *args):
            seen.append(held[0]() is not None)
            return -1 if fails else real.tq1_load_tiled_device(*args)

    def waited(stream):
        seen.append(held[0]() is not None)
        synchronize(stream)
    real = _native.lib()
    monkeypatch.setattr(torch, "empty", noted)
    monkeypatch.setattr(torch.cuda.Stream, "synchronize", waited)
    monkeypatch.setattr(_native, "lib", Library)
    if fails:
        with pytest.raises(Exception):
            module.load_tiled(*tiled)
        assert seen == [True, True]
    else:
        module.load_tiled(*tiled)
        assert seen == [True] and np.array_equal(module.blocks.cpu().numpy(), blocks)
    assert len(held) == 1
