"""Imported Node1 trees whose records name children that are not there.  The
import takes any node array; a traversal that comes to such a range ends the
ray with SQ_DEVERR_TOPOLOGY and reads nothing outside the arrays, and one that
does not come to it is not disturbed."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ERR_DEVICE = 4
TOPOLOGY = 0x4


def raw_sync(ctx):
    import sequoia_gb300 as sq
    bits = C.c_uint32()
    st = sq.load_library().sq_sync(ctx.handle, C.byref(bits))
    return st, bits.value


def device_hits(n):
    import torch
    return torch.zeros(3 * n, dtype=torch.int32, device="cuda")


def hits_of(buf):
    return buf.cpu().numpy().view(np.uint32).reshape(-1, 3)


def tree(oracle, child, fan):
    """A root of `fan` children along +z: a leaf whose triangle covers half of
    its box, an inner record that names `child`, and more such leaves."""
    tris = np.zeros((fan, 9), np.float32)
    nodes = np.zeros(1 + fan, oracle.NODE1)
    nodes[0] = ((-1, -1, 1), fan, 0, (1, 1, 2 * fan), 1)
    for j in range(fan):
        z = 2.0 * j + 1.5
        tris[j] = (-1, -1, z, 1, -1, z, -1, 1, z)
        nodes[1 + j] = ((-1, -1, z - 0.5), 1, 1, (1, 1, z + 0.5), j)
    nodes[2]["child"], nodes[2]["count"], nodes[2]["flags"] = child, 2, 0
    return nodes, tris


# bits 27-30 of a binary refill stack entry are its count, bit 31 its leaf flag
@pytest.mark.parametrize("child", [4, 1 << 27, 0x87FFFFFF, 0x90000000, 0xF8000000, 0xFFFFFFFE])
@pytest.mark.parametrize("fan", [2, 3])
@pytest.mark.parametrize("mode", ["closest", "anyhit"])
@pytest.mark.parametrize("call", ["trace", "batches"])
def test_child_index_past_the_records(ctx, oracle, child, fan, mode, call):
    nodes, tris = tree(oracle, child, fan)
    bvh = ctx.import_node1(nodes, 0, tris)

    def run(x, sched):
        rays = np.zeros((40, 8), np.float32)
        rays[:, 0:2], rays[:, 6], rays[:, 7] = x, 1.0, 100.0
        out = device_hits(len(rays))
        if call == "trace":
            ctx.trace(bvh, mode, rays=rays, hits=out, sched=sched)
        else:
            ctx.trace_batches(bvh, mode, [rays], hits=out, sched=sched)
        status = raw_sync(ctx)
        return status, hits_of(out)

    for sched in ("refill", "tiles"):
        # past the first triangle, into the box of the record
        status, _ = run(0.9, sched)
        assert status == (ERR_DEVICE, TOPOLOGY), sched
        # the first triangle ends the ray (any-hit) or culls the record
        status, got = run(-0.5, sched)
        assert status == (0, 0), sched
        assert (got[:, 0] == 0).all() and (got[:, 1].view(np.float32) == 1.5).all() and (got[:, 2] == 1 + fan).all()
    bvh.free()
