"""GPU tests of the served form (rayt_server_*): continuous batching of many
clients' frames against one shared, streamed cache.  Faulted rays restart
from the camera, so every request that ends without truncation must equal the
one-view oracle frame of its camera over a fully resident cache, alone or in
any mix."""
import threading
import time

import numpy as np
import pytest

import rayt_gb300 as R

pytestmark = pytest.mark.gpu

SIZES = [(96, 64), (160, 90), (33, 17), (128, 128), (64, 48)]


def _cam(a, v=0):
    return [a, -20.0 - 5 * (v % 3), 0.0, 0.5 - 0.6 * np.sin(np.radians(a)), 0.72,
            0.5 + 0.6 * np.cos(np.radians(a)), 60.0]


def _matrix(cam, w, h):
    return R.Camera(cam[0], cam[1], cam[2], cam[3:6], cam[6], w / h).view_proj_inv()


_REF = {}


def _resident(trees, w, h, m):
    """The oracle's one-view frame over the whole tree in the cache."""
    from oracle import oracle as O
    key = (w, h, np.asarray(m, np.float32).tobytes())
    if key not in _REF:
        sc = O.OracleScene(trees["terrain8s"], 0, w, h)
        _, img = sc.render(m)
        sc.close()
        _REF[key] = img
    return _REF[key]


def _server(trees, max_blocks=640, **kw):
    ld = R.StoredOctreeLoader(trees["terrain8s"])
    cm = R.GPUOctreeCacheManager(max_blocks, ld)
    cm.InitialFillCache()
    args = dict(max_clients=8, framebuffer_bytes=16 << 20, max_rays_in_flight=1 << 20, max_passes=32)
    args.update(kw)
    return ld, cm, R.RenderServer(cm, **args)


def test_served_alone_and_mixed_equal_resident_oracle(trees):
    frames = 4
    mats = {v: [_matrix(_cam(40.0 * f + 70 * v, v), w, h) for f in range(frames)] for v, (w, h) in enumerate(SIZES)}
    # alone: one client at a time
    alone = {}
    for v, (w, h) in enumerate(SIZES):
        ld, cm, srv = _server(trees)
        c = srv.add_client(w, h)
        for f in range(frames):
            info = srv.wait(srv.submit(c, mats[v][f]))
            assert not info["truncated"]
            alone[v, f] = srv.read_image(c)
        srv.close()
    # mixed: all clients submit together; frames of different clients share ticks
    ld, cm, srv = _server(trees)
    ids = [srv.add_client(w, h) for w, h in SIZES]
    for f in range(frames):
        reqs = [srv.submit(ids[v], mats[v][f]) for v in range(len(SIZES))]
        for v, r in enumerate(reqs):
            info = srv.wait(r)
            assert not info["truncated"] and info["client"] == ids[v]
            img = srv.read_image(ids[v])
            np.testing.assert_array_equal(img, alone[v, f], err_msg="client %d frame %d" % (v, f))
            w, h = SIZES[v]
            np.testing.assert_array_equal(img, _resident(trees, w, h, mats[v][f]), err_msg="oracle %d %d" % (v, f))
    st = srv.stats()
    assert st["completed"] == frames * len(SIZES)
    assert st["faults"] > 0  # blocks were streamed while the frames shared ticks
    assert st["ticks"] < frames * sum(1 for _ in SIZES) * 3  # frames shared ticks


def test_served_scheduler_thread_and_concurrent_submitters(trees):
    ld, cm, srv = _server(trees, deliver_to_host=True)
    ids = [srv.add_client(w, h) for w, h in SIZES]
    srv.start()
    results = {}

    def client(v):
        w, h = SIZES[v]
        for f in range(3):
            m = _matrix(_cam(33.0 * f + 50 * v, v), w, h)
            info = srv.wait(srv.submit(ids[v], m), timeout=120)
            results[v, f] = (info, srv.host_image(ids[v]).copy(), m)

    threads = [threading.Thread(target=client, args=(v,)) for v in range(len(SIZES))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    srv.stop()
    assert len(results) == 3 * len(SIZES)
    for (v, f), (info, img, m) in results.items():
        assert info["done_s"] >= info["admit_s"] >= info["submit_s"]
        if not info["truncated"]:
            w, h = SIZES[v]
            np.testing.assert_array_equal(img, _resident(trees, w, h, m), err_msg="client %d frame %d" % (v, f))


def test_served_delivery_through_client_changes(trees):
    """Host delivery while clients come and go: frames of two clients are
    delivered (their copies overlapping the next ticks), one client is
    removed right after its last frame and a client of another size takes
    its slot; every delivered image equals the resident oracle frame."""
    ld, cm, srv = _server(trees, max_blocks=0, deliver_to_host=True)  # resident: no request truncates
    a = srv.add_client(96, 64)
    b = srv.add_client(160, 90)
    for f in range(3):
        ma, mb = _matrix(_cam(25.0 * f, 0), 96, 64), _matrix(_cam(25.0 * f + 90, 1), 160, 90)
        ra, rb = srv.submit(a, ma), srv.submit(b, mb)
        srv.wait(ra)
        np.testing.assert_array_equal(srv.host_image(a), _resident(trees, 96, 64, ma), err_msg="a %d" % f)
        srv.wait(rb)
        np.testing.assert_array_equal(srv.host_image(b), _resident(trees, 160, 90, mb), err_msg="b %d" % f)
    srv.remove_client(b)
    c = srv.add_client(128, 128)
    for f in range(2):
        ma, mc = _matrix(_cam(40.0 * f + 10, 0), 96, 64), _matrix(_cam(40.0 * f + 200, 2), 128, 128)
        ra, rc = srv.submit(a, ma), srv.submit(c, mc)
        srv.wait(rc)
        np.testing.assert_array_equal(srv.host_image(c), _resident(trees, 128, 128, mc), err_msg="c %d" % f)
        srv.wait(ra)
        np.testing.assert_array_equal(srv.host_image(a), _resident(trees, 96, 64, ma), err_msg="a' %d" % f)
    assert srv.stats()["completed"] == 10
    srv.close()


@pytest.mark.parametrize("max_blocks", [0, 640])
def test_served_delivery_in_groups(trees, max_blocks):
    """A tick large enough to be traced group by group (three frames of a little
    over 2^22 pixels each): the frames of all but the last group go to the host
    beside the groups after them, unless a ray of theirs faulted; every
    delivered image equals the resident oracle frame."""
    w, h, frames = 2304, 1824, 3
    pixels = 3 * w * h
    ld, cm, srv = _server(trees, max_blocks=max_blocks, deliver_to_host=True, framebuffer_bytes=4 * pixels,
                          max_rays_in_flight=pixels)
    ids = [srv.add_client(w, h) for _ in range(3)]
    for f in range(frames):
        mats = [_matrix(_cam(70.0 * v + 15.0 * (f % 2), v), w, h) for v in range(3)]
        reqs = [srv.submit(c, m) for c, m in zip(ids, mats)]
        for r in reqs:
            assert not srv.wait(r)["truncated"]
        for v, (c, m) in enumerate(zip(ids, mats)):
            np.testing.assert_array_equal(srv.host_image(c), _resident(trees, w, h, m), err_msg="%d %d" % (v, f))
    srv.close()


@pytest.mark.parametrize("requests", [1, 2, 3])
def test_served_delivery_under_backlog(trees, requests):
    """Requests that wait behind a tick (frames then go through the stages beside
    the next tick) and none (frames go straight from the framebuffers, in groups
    where there are many rays): each client's last image is the resident oracle's."""
    sizes = [(1280, 720), (96, 64), (1024, 1024)]
    pixels = sum(w * h + 64 for w, h in sizes)
    ld, cm, srv = _server(trees, max_blocks=0, deliver_to_host=True, framebuffer_bytes=4 * pixels,
                          max_rays_in_flight=pixels)
    ids = [srv.add_client(w, h) for w, h in sizes]
    for f in range(2):
        mats = [[_matrix(_cam(70.0 * v + 25.0 * k + 40.0 * f, v), w, h) for k in range(requests)]
                for v, (w, h) in enumerate(sizes)]
        for r in [srv.submit(c, m) for k in range(requests) for c, m in zip(ids, (x[k] for x in mats))]:
            assert not srv.wait(r)["truncated"]
        for v, (c, (w, h)) in enumerate(zip(ids, sizes)):
            np.testing.assert_array_equal(srv.host_image(c), _resident(trees, w, h, mats[v][-1]), err_msg="%d %d" % (v, f))
    srv.close()


def test_served_admission_limits(trees):
    # framebuffer memory admits clients: 2 frames of 128x128 fit, a third does not
    ld, cm, srv = _server(trees, framebuffer_bytes=2 * 128 * 128 * 4)
    a = srv.add_client(128, 128)
    b = srv.add_client(128, 128)
    with pytest.raises(R.RaytError):
        srv.add_client(128, 128)
    srv.remove_client(b)
    c = srv.add_client(64, 64)
    # ray-record capacity admits requests: one 128x128 request at a time
    srv.close()
    ld, cm, srv = _server(trees, max_rays_in_flight=128 * 128)
    a = srv.add_client(128, 128)
    b = srv.add_client(128, 128)
    ra = srv.submit(a, _matrix(_cam(10.0), 128, 128))
    rb = srv.submit(b, _matrix(_cam(100.0), 128, 128))
    ia, ib = srv.wait(ra), srv.wait(rb)
    assert ib["admit_s"] >= ia["done_s"] - 1e-3  # b waited for a's records
    # one request per client at a time, in order
    r1 = srv.submit(a, _matrix(_cam(20.0), 128, 128))
    r2 = srv.submit(a, _matrix(_cam(30.0), 128, 128))
    i2 = srv.wait(r2)
    i1 = srv.wait(r1)
    assert i2["admit_s"] >= i1["done_s"] - 1e-3
    np.testing.assert_array_equal(srv.read_image(a), _resident(trees, 128, 128, _matrix(_cam(30.0), 128, 128)))


def test_served_pass_cap_truncates(trees):
    ld, cm, srv = _server(trees, max_blocks=60, max_passes=1)
    c = srv.add_client(160, 90)
    info = srv.wait(srv.submit(c, _matrix(_cam(0.0), 160, 90)))
    assert info["passes"] == 1
    assert info["truncated"] == 1
    img = srv.read_image(c)
    assert img[..., 3].min() == 255  # every pixel was written


def _mix_under_eviction(trees, max_blocks, sizes, mats, frames):
    """Requests compared (alone = mixed = oracle) and blocks uploaded, for one
    shared cache size."""
    alone = {}
    for v, (w, h) in enumerate(sizes):
        ld, cm, srv = _server(trees, max_blocks=max_blocks)
        c = srv.add_client(w, h)
        for f in range(frames):
            info = srv.wait(srv.submit(c, mats[v][f]))
            alone[v, f] = (info["truncated"], srv.read_image(c))
        srv.close()
    ld, cm, srv = _server(trees, max_blocks=max_blocks)
    ids = [srv.add_client(w, h) for w, h in sizes]
    compared = 0
    for f in range(frames):
        reqs = [srv.submit(ids[v], mats[v][f]) for v in range(len(sizes))]
        for v, r in enumerate(reqs):
            info = srv.wait(r)
            if info["truncated"] or alone[v, f][0]:
                continue
            img = srv.read_image(ids[v])
            np.testing.assert_array_equal(img, alone[v, f][1], err_msg="cache %d client %d frame %d" % (max_blocks, v, f))
            w, h = sizes[v]
            np.testing.assert_array_equal(img, _resident(trees, w, h, mats[v][f]),
                                          err_msg="cache %d oracle %d %d" % (max_blocks, v, f))
            compared += 1
    uploaded = cm.stats()["uploaded_blocks"]
    srv.close()
    return compared, uploaded


def test_served_mix_under_eviction_equals_alone(trees):
    """A shared cache smaller than the tree (790 blocks): the mixed clients'
    blocks evict one another from the one LRU, and every request that ends
    without truncation still has the image it has alone and the oracle's
    resident one-view image (restart semantics).  Cache sizes are tried from
    large to small until one both evicts (more blocks uploaded than it holds)
    and leaves at least two requests untruncated; every untruncated request of
    every size tried is checked."""
    frames = 5
    sizes = SIZES[:3]
    mats = {v: [_matrix(_cam(72.0 * f + 40 * v, v), w, h) for f in range(frames)] for v, (w, h) in enumerate(sizes)}
    seen = []
    for max_blocks in (600, 450, 330, 240):
        compared, uploaded = _mix_under_eviction(trees, max_blocks, sizes, mats, frames)
        seen.append((max_blocks, compared, uploaded))
        if compared >= 2 and uploaded > max_blocks:
            return
    raise AssertionError("no cache size both evicted and kept two requests untruncated: %s" % seen)


def test_served_image_stays_the_last_finished_frame(trees):
    """Two clients in one tick: the first looks past the scene and is done, and
    its large frame is on its way to the host through the ticks after it; the
    second's copy is queued behind it and its rays fault for some ticks.  The
    second's host image stays its last finished frame until the request is
    done, whatever those ticks have done to the counts by then."""
    import torch
    big, w, h = 8192, 160, 90
    ld, cm, srv = _server(trees, max_blocks=400, max_clients=2, deliver_to_host=True,
                          framebuffer_bytes=4 * (big * big + w * h + 64), max_rays_in_flight=big * big + w * h)
    a, b = srv.add_client(big, big), srv.add_client(w, h)
    away = R.Camera(0.0, 80.0, 0.0, (0.5, 3.0, 0.5), 40.0, 1.0).view_proj_inv()
    before, after = _matrix(_cam(0.0), w, h), _matrix(_cam(80.0), w, h)
    assert not srv.wait(srv.submit(b, before))["truncated"]
    np.testing.assert_array_equal(srv.host_image(b), _resident(trees, w, h, before))
    ra, rb = srv.submit(a, away), srv.submit(b, after)
    assert srv.step() == 1  # a
    assert srv.step() == 0  # only carries b's rays
    torch.cuda.synchronize()  # every copy queued so far
    np.testing.assert_array_equal(srv.host_image(b), _resident(trees, w, h, before))
    assert not srv.wait(rb)["truncated"] and not srv.wait(ra)["truncated"]
    np.testing.assert_array_equal(srv.host_image(b), _resident(trees, w, h, after))
    assert (srv.host_image(a) == (0, 216, 255, 255)).all()
    srv.close()


def _late_blocks(loader, resident):
    """Blocks below a child of the root block that the initial fill of a cache of
    `resident` blocks does not load: none of them is requested before its parent
    was."""
    info = loader.info
    links = loader.LoadBlock(info.root_block_index)[1][:4 * info.nodes_in_block].view(np.uint32)
    named = [int(l) >> 11 for l in links if (int(l) & 0x1FF) > 0x100]
    loaded = set(list(dict.fromkeys(named))[:resident - 1])
    parents = [loader.LoadBlock(b)[0].parent_block_index for b in range(info.blocks_count)]
    below_root = {b for b, p in enumerate(parents) if p == info.root_block_index}
    return [b for b, p in enumerate(parents) if p in below_root - loaded]


@pytest.mark.parametrize("mode", ["mapped", "read"])
def test_served_request_survives_a_failed_tick(trees, tmp_path, monkeypatch, mode):
    """A block that cannot be read fails the tick that asks for it, in the middle
    of two requests, some of whose rays are carried over; once the file is whole
    again both end with the image of a run in which nothing failed."""
    monkeypatch.setenv("RAYT_BLOCK_IO", mode)
    path, resident = str(tmp_path / "scene.tree"), 250
    with open(trees["terrain8s"], "rb") as f:
        whole = f.read()
    with open(path, "wb") as f:
        f.write(whole)
    ld = R.StoredOctreeLoader(path)
    info = ld.info
    late = _late_blocks(ld, resident)
    cm = R.GPUOctreeCacheManager(resident, ld)
    cm.InitialFillCache()
    assert cm.stats()["mapped"] == (mode == "mapped")
    srv = R.RenderServer(cm, max_clients=2, framebuffer_bytes=1 << 20, max_rays_in_flight=1 << 18, max_passes=32)
    sizes = [(160, 90), (33, 17)]
    ids = [srv.add_client(w, h) for w, h in sizes]
    mats = [_matrix(_cam(0.0 + 40 * v), w, h) for v, (w, h) in enumerate(sizes)]
    reqs = [srv.submit(c, m) for c, m in zip(ids, mats)]
    with open(path, "r+b", buffering=0) as f:
        for b in late:  # a root count of zero: the record is refused
            f.seek(info.header_bytes + info.block_stride * b + 8)
            f.write(b"\0\0\0\0")
    steps = 0
    with pytest.raises(R.RaytError):
        while steps < 32:
            steps += srv.step() >= 0
    assert steps >= 1 and srv.stats()["completed"] < 2
    with pytest.raises(R.RaytError):  # and again
        srv.step()
    with open(path, "r+b", buffering=0) as f:
        f.write(whole)
    for v, ((w, h), c, r, m) in enumerate(zip(sizes, ids, reqs, mats)):
        assert not srv.wait(r)["truncated"]
        np.testing.assert_array_equal(srv.read_image(c), _resident(trees, w, h, m), err_msg="client %d" % v)
    assert srv.stats()["completed"] == 2
    srv.close()


def test_served_tick_does_not_wait_for_copies_from_framebuffers(trees):
    """A large frame goes to the host straight from its framebuffer, which reads
    no stage: a smaller frame that ends in a later tick goes to its stage, and
    the tick after that, which carries the rays of others, ends while the large
    copy (3 ms) is under way: one of a few such ticks at least takes less than
    1 ms (they take 0.1)."""
    bw, bh, w, h, small = 16384, 8192, 160, 90, 3
    pixels = bw * bh + small * (w * h + 64)
    ld, cm, srv = _server(trees, max_blocks=640, deliver_to_host=True, framebuffer_bytes=4 * pixels,
                          max_rays_in_flight=pixels)
    a, ids = srv.add_client(bw, bh), [srv.add_client(w, h) for _ in range(small)]
    away = R.Camera(0.0, 80.0, 0.0, (0.5, 3.0, 0.5), 40.0, 1.0).view_proj_inv()
    ticks = []
    for f in range(6):
        mats = [_matrix(_cam(80.0 * f + 55.0 * v, v), w, h) for v in range(small)]
        done = srv.stats()["completed"]
        reqs = [srv.submit(a, away)] + [srv.submit(c, m) for c, m in zip(ids, mats)]
        left = small + 1 - srv.step()
        staged = False
        while left > 0:
            t0 = time.perf_counter()
            n = srv.step()
            if srv.stats()["completed"] != done:
                break
            if staged:
                ticks.append(time.perf_counter() - t0)
            staged = n > 0
            left -= n
        srv.wait(reqs[0])
        for c, r, m in zip(ids, reqs[1:], mats):
            if not srv.wait(r)["truncated"]:
                np.testing.assert_array_equal(srv.host_image(c), _resident(trees, w, h, m), err_msg="frame %d" % f)
    assert min(ticks) < 1e-3
    srv.close()
