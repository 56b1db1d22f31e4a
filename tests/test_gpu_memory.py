"""What a handle, a batch and a server allocate: the parts that wide bonds share
come when a launch can have such a bond, not with the object, so an object that
never gets there takes its state and one workspace per CTA (32 bytes for each
entry of theta in double-float)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CAP = 512
WORKSPACE = 2 * 4 * CAP * CAP * 16  # theta and the vectors of a CTA, double-float
SLACK = 64 << 20  # context, pools and small buffers


def _used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_parts_come_with_wide_bonds(pkg):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pkg.MPS.new_qubits(4, None, "df").apply_unitary2(0, np.eye(4))  # module loading
    tr = pkg.Trunc.both(CAP, 1e-10)
    n = 20
    state = 2 * CAP * CAP * 16 * n
    at = _used()
    m = pkg.MPS.new_qubits(n, tr, "df")
    assert _used() - at < state + 1.2 * WORKSPACE + SLACK
    at = _used()
    b = pkg.Batch([n] * 4, [tr] * 4, "df")
    ctas = min(sms, 4 * n // 2)
    assert _used() - at < 4 * state + 1.2 * ctas * WORKSPACE + SLACK
    at = _used()
    layer = pkg.gen_layer(1, 0, 0, n, 0.0)
    m.apply_bilayer(*layer)
    b.step([0, 1], [layer] * 2)
    # narrow bonds need none; the handle's disjoint gates take a workspace each
    assert _used() - at < 1.2 * (n // 2) * WORKSPACE + SLACK
    assert b.svals(0, n // 2 - 1).tolist() == m.svals(n // 2 - 1).tolist()
    assert b.device_status() == 0 and m.device_status() == 0


def test_server_with_an_arena_that_leaves_room_for_workspaces_only(pkg):
    """A large arena beside the classes' workspaces: created as long as both fit."""
    import torch
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    s = pkg.Server(int(free - 1.3 * sms * WORKSPACE - (2 << 30)), 8, "df", CAP, 20)
    del s
