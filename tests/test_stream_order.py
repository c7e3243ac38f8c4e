"""Encode returns with its kernels in flight. What the caller may do then: record
encodes into a graph, whatever stream the last encode was on and wherever the
frame lies; read, or upload a ring table, after encodes that had nothing to add on
another stream; read on a stream whose handle was the encodes', or after an encode
that failed; change a frame in pinned memory."""
import ctypes as C

import numpy as np
import pytest

from stargaze_b200 import abi
from stargaze_b200 import workloads as W
from stargaze_b200._lib import StargazeError, check
from stargaze_b200.pathtracer import PathTracer

pytestmark = pytest.mark.gpu


def tracer_of(wl, spp=4, integrator="wavefront", **options):
    o = W.render_options(wl, spp, noise_seed=3)
    for name, value in options.items():
        setattr(o, name, value)
    t = PathTracer((wl.width, wl.height), o)
    W.upload_workload(t, wl)
    t.set_integrator(integrator)
    return t


def encode_view(t, view, stream):
    check(t._lib.sg_encode(t.handle, C.byref(view), C.c_void_p(stream)), t.handle)


def pin_bodies(view):
    """The view's bodies moved to pinned memory; returns that memory."""
    import torch

    size = view.n_bodies * C.sizeof(abi.Sphere)
    held = torch.empty(size, dtype=torch.uint8).pin_memory()
    C.memmove(held.data_ptr(), view.bodies, size)
    view.bodies = C.cast(C.c_void_p(held.data_ptr()), C.POINTER(abi.Sphere))
    return held


@pytest.mark.parametrize("pinned", [False, True], ids=["pageable", "pinned"])
def test_encode_records_into_a_graph(pinned):
    """The megakernel's encode on a capturing stream that is not the last
    encode's, then a launch of the graph: as two encodes. The image is read, and
    a ring table uploaded, as after any encode."""
    import torch

    wl = W.rings_1080p(64, 48)
    plain = tracer_of(wl, integrator="megakernel")
    for _ in range(2):
        plain.encode(wl.frame)
    t = tracer_of(wl, integrator="megakernel")
    view = wl.frame.view()
    held = pin_bodies(view) if pinned else None
    encode_view(t, view, 0)
    torch.cuda.synchronize()
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=side):
        encode_view(t, view, side.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    assert t.samples() == plain.samples()
    assert np.array_equal(t.read_pixels(), plain.read_pixels())
    t.upload_ring_profile(0, wl.ring_tables[0])
    t.encode(wl.frame)
    assert np.isfinite(t.read_pixels()).all()
    del held
    graph.reset()
    t.close()
    plain.close()


def delayed_encodes(t, wl, stream):
    """Three dispatches on `stream`, held back there for tens of milliseconds."""
    import torch

    with torch.cuda.stream(stream):
        torch.cuda._sleep(100_000_000)
    for _ in range(3):
        t.encode(wl.frame, stream)


def image_of(wl, **options):
    t = tracer_of(wl, **options)
    for _ in range(3):
        t.encode(wl.frame)
    image = t.read_pixels()
    t.close()
    assert np.abs(image[:, :3]).sum() > 0
    return image


@pytest.mark.parametrize("upload", [False, True], ids=["read", "upload"])
def test_an_encode_with_nothing_to_add_leaves_the_order(upload):
    """The sample limit is reached on one stream, the next encode is on another:
    what follows there still waits for the samples."""
    import torch

    wl = W.rings_1080p(640, 360)
    expected = image_of(wl, sample_limit=12)
    t = tracer_of(wl, sample_limit=12)
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    delayed_encodes(t, wl, first)
    t.encode(wl.frame, second)
    assert t.samples() == 12
    if upload:  # the dispatches in flight read the table they were given
        t.upload_ring_profile(0, np.zeros(512, np.float32))
    assert np.array_equal(t.read_pixels(second), expected)
    t.close()


def test_one_handle_for_two_streams():
    """cudaStreamPerThread in two threads: the same handle, two streams."""
    import threading

    import torch

    per_thread = 2
    wl = W.rings_1080p(640, 360)
    plain, t = tracer_of(wl), tracer_of(wl)
    for _ in range(4):
        plain.encode(wl.frame)
    t.encode(wl.frame)  # allocates
    encoded, read = threading.Event(), threading.Event()

    def encodes():
        delayed_encodes(t, wl, torch.cuda.ExternalStream(per_thread))
        encoded.set()
        read.wait()

    thread = threading.Thread(target=encodes)
    thread.start()
    encoded.wait()
    image = t.read_pixels(per_thread)
    read.set()
    thread.join()
    assert np.array_equal(image, plain.read_pixels())
    plain.close()
    t.close()


def test_a_failed_encode_is_waited_for_too():
    """An encode that fails for want of checkpoint memory has copied its frame: reading on
    another stream comes after that copy."""
    import torch

    wl = W.rings_1080p(64, 48)
    t = tracer_of(wl)
    t.encode(wl.frame)
    before = t.read_pixels()
    t.set_checkpoints(1, 64, 1)  # a byte holds no record
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(first):
        torch.cuda._sleep(100_000_000)
    with pytest.raises(StargazeError) as e:
        t.encode(wl.frame, first)
    assert e.value.status == abi.SG_ERR_OOM
    assert np.array_equal(t.read_pixels(second), before)
    assert first.query()
    t.close()


@pytest.mark.parametrize("integrator", ["megakernel", "wavefront"])
def test_a_pinned_frame_may_change_once_encode_has_returned(integrator):
    """And encode returns before the GPU gets to the frame's copy."""
    import torch

    wl = W.rings_1080p(64, 48)
    plain, t = tracer_of(wl, integrator=integrator), tracer_of(wl, integrator=integrator)
    for _ in range(2):
        plain.encode(wl.frame)
    t.encode(wl.frame)  # allocates
    torch.cuda.synchronize()
    view, stream = wl.frame.view(), torch.cuda.Stream()
    held = pin_bodies(view)
    with torch.cuda.stream(stream):
        torch.cuda._sleep(200_000_000)
    asleep = stream.record_event()
    encode_view(t, view, stream.cuda_stream)
    assert not asleep.query()
    held.zero_()
    assert np.array_equal(t.read_pixels(stream), plain.read_pixels())
    plain.close()
    t.close()
