"""The captured binary16 forward: the values of the operator-by-operator one, and handles a caller keeps stay as they were."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_captured_forward_keeps_values_and_handles():
    import lightnet_b200 as ln
    from lightnet_b200 import synth, zoo
    be = ln.B200Backend(0)
    nets = [ln.GpuExecutableNetwork(be, zoo.yolov3_tiny_cfg(160, 96), 2, ln.LN_F16) for _ in range(2)]
    blob = synth.he_weights(nets[0].layers(), 3)
    for net in nets:
        net.load_weights(blob)
    nets[1].set_cuda_graph(False)
    images = [synth.uniform_images(2, 3, 96, 160, s) for s in range(6)]

    def heads(net):
        return [be.download_f32(net.head(k)) for k in range(net.num_heads())]

    want = []
    for x in images:
        nets[1].forward(x)
        want.append(heads(nets[1]))
    kept, kept_layer = None, None
    for i, x in enumerate(images):  # eager, captured, replayed, (two with handles kept across them), replayed
        nets[0].forward(x)
        assert nets[0].debug_replays() == [0, 1, 2, 2, 2, 3][i]
        for got, ref in zip(heads(nets[0]), want[i]):
            np.testing.assert_array_equal(got, ref)
        if i == 2:
            kept, kept_layer = nets[0].head(0), nets[0].layer_output(4)
            before = be.download_f16(kept_layer)
        if i in (3, 4):  # forwards since then left the kept tensors alone
            np.testing.assert_array_equal(be.download_f32(kept), want[2][0])
            np.testing.assert_array_equal(be.download_f16(kept_layer), before)
        if i == 4:
            del kept, kept_layer
    nets[0].load_weights(blob * np.float32(0.5))  # new weights: nothing of the old graph is left
    nets[1].load_weights(blob * np.float32(0.5))
    for x in images[:3]:
        for net in nets:
            net.forward(x)
        for got, ref in zip(heads(nets[0]), heads(nets[1])):
            np.testing.assert_array_equal(got, ref)
    assert nets[0].debug_replays() == 5 and nets[1].debug_replays() == 0
    del nets
    be.close()


def test_a_capture_that_failed_is_tried_again():
    import lightnet_b200 as ln
    from lightnet_b200 import synth, zoo
    be = ln.B200Backend(0)
    net = ln.GpuExecutableNetwork(be, zoo.yolov3_tiny_cfg(160, 96), 2, ln.LN_F16)
    net.load_weights(synth.he_weights(net.layers(), 3))
    x = synth.uniform_images(2, 3, 96, 160, 4)
    net.forward(x)
    want = be.download_f32(net.head(0))
    be.debug_fail_alloc(12)  # in the middle of the captured layers
    net.forward(x)
    assert net.debug_replays() == 0
    np.testing.assert_array_equal(be.download_f32(net.head(0)), want)
    net.forward(x)
    assert net.debug_replays() == 1
    np.testing.assert_array_equal(be.download_f32(net.head(0)), want)
    del net
    be.close()


def test_first_forward_out_of_memory_then_capture_out_of_memory():
    """A first forward that runs out of memory half way, then a capture that does: the forwards after them compute with packed weights."""
    import lightnet_b200 as ln
    from lightnet_b200 import synth, zoo
    be = ln.B200Backend(0)
    cfg = zoo.yolov3_tiny_cfg(160, 96)
    blob = synth.he_weights(ln.GpuExecutableNetwork(be, cfg, 2, ln.LN_F16).layers(), 3)
    x = synth.uniform_images(2, 3, 96, 160, 4)

    def heads(net):
        net.forward(x)
        return [be.download_f32(net.head(k)) for k in range(net.num_heads())]

    ref_net = ln.GpuExecutableNetwork(be, cfg, 2, ln.LN_F16)
    ref_net.load_weights(blob)
    ref_net.set_cuda_graph(False)
    want = heads(ref_net)
    garbage = be.upload_f32((1, 1, 2048, 4096), np.full(2048 * 4096, 1e3, np.float32))  # what a block of the pool holds before it is packed
    del garbage
    refused = 0
    for first in range(20, 60, 6):
        for second in range(first, 60, 6):
            net = ln.GpuExecutableNetwork(be, cfg, 2, ln.LN_F16)
            net.load_weights(blob)
            for n in (first, second):
                be.debug_fail_alloc(n)
                try:
                    got = heads(net)
                except ln.BackendError as e:
                    assert "refused" in str(e)
                    refused += 1
                else:
                    for g, w in zip(got, want):
                        np.testing.assert_array_equal(g, w)
            be.debug_fail_alloc(0)
            for _ in range(3):
                for g, w in zip(heads(net), want):
                    np.testing.assert_array_equal(g, w)
            del net
    assert refused > 0
    be.close()


def test_kept_handle_and_no_room_for_a_second_set_of_outputs():
    """A forward that may not replay the graph (a head of it is kept) and runs out of memory gives the graph's tensors back and succeeds."""
    import lightnet_b200 as ln
    from lightnet_b200 import synth, zoo
    be = ln.B200Backend(0)
    cfg = zoo.yolov3_tiny_cfg(160, 96)
    nets = [ln.GpuExecutableNetwork(be, cfg, 2, ln.LN_F16) for _ in range(2)]
    for net in nets:
        net.load_weights(synth.he_weights(net.layers(), 3))
    nets[1].set_cuda_graph(False)
    x = [synth.uniform_images(2, 3, 96, 160, s) for s in range(2)]

    def heads(net, x):
        net.forward(x)
        return [be.download_f32(net.head(k)) for k in range(net.num_heads())]

    want = [heads(nets[1], v) for v in x]
    for n in (1, 2, 11):
        for _ in range(3):  # operator by operator, captured, replayed
            heads(nets[0], x[0])
        kept = nets[0].head(0)
        be.debug_fail_alloc(n)
        for g, w in zip(heads(nets[0], x[1]), want[1]):
            np.testing.assert_array_equal(g, w)
        be.debug_fail_alloc(0)
        np.testing.assert_array_equal(be.download_f32(kept), want[0][0])
        del kept
    del nets, net
    be.close()
