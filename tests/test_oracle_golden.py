"""CPU: the oracle restatements AND the product's host code against fixtures produced by the reference itself
(tests/golden/*.json, generated by oracle/make_golden.py).  Mirrors the reference's own pins:
tests/test_worker_distributed_model_shard.py:299-344,436-527, tests/test_common_serialization.py:20-107,
tests/test_worker_distributed_kv_cache.py:218-290,329-343,397-412."""
import json

import numpy as np
import pytest
import torch

import dgi_b200  # noqa: F401
from dgi_b200.common import data_structures as ds
from dgi_b200.common import serialization as ser
from dgi_b200.worker.distributed import kv_cache as kv
from dgi_b200.worker.distributed import model_shard as ms
from oracle import host_logic as H
from oracle import llama_ref as L


# ---- layer ranges ----------------------------------------------------------------------------------------
def test_layer_ranges_match_reference(golden):
    g = golden("host_logic.json")["layer_ranges"]
    for key, want in g.items():
        total, n = map(int, key.split("/"))
        assert [list(H.layer_range(total, n, i)) for i in range(n)] == want
        assert [list(ms.get_layer_range_for_worker(total, n, i)) for i in range(n)] == want


def test_layer_ranges_reference_test_vectors():
    # the literal expectations of the reference's tests (test_worker_distributed_model_shard.py:299-344)
    assert [ms.get_layer_range_for_worker(32, 4, i) for i in range(4)] == [(0, 8), (8, 16), (16, 24), (24, 32)]
    assert [ms.get_layer_range_for_worker(10, 3, i) for i in range(3)] == [(0, 4), (4, 7), (7, 10)]
    rs = [ms.get_layer_range_for_worker(5, 10, i) for i in range(10)]
    assert rs[:5] == [(i, i + 1) for i in range(5)] and all(a == b for a, b in rs[5:])
    cover = [ms.get_layer_range_for_worker(80, 5, i) for i in range(5)]
    assert cover[0][0] == 0 and cover[-1][1] == 80 and all(cover[i][1] == cover[i + 1][0] for i in range(4))


def test_device_map_keys(golden):
    g = golden("host_logic.json")
    dm = ms._create_device_map_for_layers(None, 2, 5, "cuda:0", include_embeddings=True, include_lm_head=True)
    assert [list(kv_) for kv_ in dm.items()] == g["device_map_2_5_first_last"]
    dm2 = ms._create_device_map_for_layers(None, 0, 2, "cpu")
    assert [list(kv_) for kv_ in dm2.items()] == g["device_map_0_2_plain"]


def test_shard_plans_match_reference(golden):
    plans = golden("host_logic.json")["shard_plans"]
    shapes = {"8b": L.LLAMA3_8B, "70b": L.LLAMA3_70B, "tiny": L.TINY}
    for name, entry in plans.items():
        cfg = L.RefConfig(**shapes[name])
        loader = ms.ShardedModelLoader(name, config=cfg)
        info = loader.analyze_model()
        for k, v in entry["info"].items():
            assert info[k] == pytest.approx(v) if isinstance(v, float) else info[k] == v
        for mems, want in entry["plans"].items():
            mems = json.loads(mems)
            if isinstance(want, dict):
                with pytest.raises(ValueError) as ei:
                    loader.create_shard_plan(mems)
                assert str(ei.value) == want["ValueError"]
            else:
                assert [list(p) for p in loader.create_shard_plan(mems)] == want


# ---- hashes / headers --------------------------------------------------------------------------------------
def test_prefix_hash(golden):
    g = golden("host_logic.json")
    for toks, want in g["prefix_hashes"].items():
        toks = json.loads(toks)
        assert H.prefix_hash(toks) == want
        assert ds.compute_prefix_hash(toks) == want
        assert kv.DistributedKVCacheManager.compute_prefix_hash(None, toks) == want
    assert ds.compute_prefix_hash([1, 2, 3, 4, 5]) == "74f81fe167d99b4c"  # as the reference gives it
    assert g["prefix_hash_raises_for_256"]
    with pytest.raises(ValueError):
        ds.compute_prefix_hash([256])
    assert len(ds.compute_prefix_hash_wide([128000, 5])) == 16


def test_stream_headers(golden):
    for key, want in golden("host_logic.json")["stream_headers"].items():
        shape, dt = json.loads(key)
        assert H.stream_header(tuple(shape), dt).hex() == want
        buf = ser.StreamingTensorBuffer()
        hdr = buf.write_header(tuple(shape), dt)
        assert hdr.hex() == want
        back = buf.read_header(hdr)
        assert back["shape"] == tuple(shape)
    assert H.stream_header((2, 3), "bfloat16").hex() == "02000000" "0200000000000000" "0300000000000000" "02"


def test_misc_host_numbers(golden):
    g = golden("host_logic.json")
    assert ds.estimate_kv_cache_size(32, 8, 128, 2048, 64) == g["estimate_kv_cache_size_32_8_128_2048_64"]
    mgr = kv.DistributedKVCacheManager(num_layers=1, num_heads=8, head_dim=128, gpu_cache_blocks=4, device="cpu")
    assert mgr.cpu_cache_max_items == g["cpu_cache_max_items_16g_8h_128d"] == 262144
    assert sorted(mgr.get_stats().keys()) == g["manager_stats_keys"]
    assert sorted(kv.PagedKVCache(1, 2, 8, max_blocks=2, device="cpu").get_stats().keys()) == g["paged_stats_keys"]


# ---- allocator ---------------------------------------------------------------------------------------------
def _replay_product(max_blocks, schedule):
    cache = kv.PagedKVCache(num_layers=1, num_heads=2, head_dim=8, block_size=4, max_blocks=max_blocks, device="cpu")
    handed = []
    for op, arg in schedule:
        if op == "alloc":
            blk = cache.allocate_block(0)
            handed.append(blk.block_id if blk is not None else None)
        elif op == "free":
            if handed[arg] is not None:
                cache.free_block(handed[arg])
        elif op == "ref":
            if handed[arg] is not None and handed[arg] in cache._blocks:
                cache._blocks[handed[arg]].add_ref()
        elif op == "touch":
            cache.get_block(handed[arg])
    stats = cache.get_stats()
    stats.pop("memory_gb")
    return {"handed": handed, "free": list(cache._free_blocks), "stats": stats}


def test_allocator_schedules_bit_exact(golden):
    g = golden("allocator.json")
    for name, entry in g.items():
        if "schedule" not in entry:
            continue
        sched = [tuple(x) for x in entry["schedule"]]
        want = {k: entry[k] for k in ("handed", "free", "stats")}
        assert H.run_allocator_schedule(entry["max_blocks"], sched) == want, name
        assert _replay_product(entry["max_blocks"], sched) == want, name


def test_allocator_survey_probe(golden):
    e = golden("allocator.json")["survey_probe"]
    assert e["handed"][:3] == ["block_7", "block_6", "block_5"]
    assert e["handed"][3:9] == ["block_6", "block_4", "block_3", "block_2", "block_1", "block_0"]
    assert e["handed"][9] == "block_7" and e["stats"]["evictions"] == 1 and e["stats"]["allocations"] == 10


def test_allocate_sequence_ids(golden):
    want = golden("allocator.json")["allocate_sequence_bs16_max20"]
    pool = kv.KVCachePool(num_layers=3, num_heads=2, head_dim=8, block_size=16, max_blocks_per_layer=20, device="cpu")
    for seq_len, ids in sorted(want.items(), key=lambda kv_: int(kv_[0])):  # generation order: 1, 16, 17, 100
        blocks = pool.allocate_sequence(int(seq_len))
        assert [[b.block_id for b in layer] for layer in blocks] == ids
        assert all(len(layer) == H.blocks_for(int(seq_len), 16) for layer in blocks)
        assert kv.KVCachePool.block_table(blocks[0]) == [int(i.split("_")[1]) for i in ids[0]]


def test_freed_slot_reads_zero_and_views_alias_pool():
    cache = kv.PagedKVCache(1, 2, 8, block_size=4, max_blocks=4, device="cpu", dtype=torch.float32)
    blk = cache.allocate_block(0)
    blk.keys.fill_(3.0)
    assert cache.key_pool[blk.slot].eq(3.0).all()  # CacheBlock.keys is a view (reference kv_cache.py:184-185)
    cache.free_block(blk.block_id)
    assert cache.key_pool[blk.slot].eq(0).all()
    cache.free_block("block_999")  # unknown id: silent


def test_allocate_sequence_failure_rolls_back():
    # intended behaviour of the reference's test_allocate_sequence_failure (tests/...kv_cache.py:345-361)
    pool = kv.KVCachePool(num_layers=2, num_heads=2, head_dim=8, block_size=16, max_blocks_per_layer=2, device="cpu")
    with pytest.raises(RuntimeError, match="Failed to allocate KV-Cache for layer 0"):
        pool.allocate_sequence(100)
    assert all(c.get_stats()["free_blocks"] == 2 for c in pool._layer_caches)


# ---- serializer --------------------------------------------------------------------------------------------
_BITS = {2: torch.int16, 4: torch.int32, 8: torch.int64}


def test_serializer_matches_reference_bytes(golden):
    g = golden("serializer.json")
    for name, c in g.items():
        if "input_bits_hex" not in c:
            continue
        dt = getattr(torch, c["input_dtype"])
        es = torch.empty((), dtype=dt).element_size()
        raw = np.frombuffer(bytes.fromhex(c["input_bits_hex"]), dtype=np.dtype(f"i{es}")).copy()
        t = torch.from_numpy(raw).view(dt).reshape(c["shape"])
        data, shape, dtype_str = ser.TensorSerializer.serialize(t)
        assert data.hex() == c["bytes_hex"] and list(shape) == c["shape"] and dtype_str == c["dtype_str"], name
        assert ser.serialize_tensor(t) == c["envelope"], name
        back = ser.deserialize_tensor(c["envelope"])
        assert str(back.dtype) == "torch." + c["roundtrip_dtype"]
        got = back.to(torch.float64).flatten().tolist()
        assert all((a == b) or (a != a and b != b) for a, b in zip(got, c["roundtrip_values"])), name
    arr = np.arange(6, dtype=np.float32).reshape(2, 3)
    data, shape, dtype_str = ser.TensorSerializer.serialize(arr)
    assert data.hex() == g["numpy_f32_2x3"]["bytes_hex"] and dtype_str == "float32"
    with pytest.raises(TypeError) as ei:
        ser.TensorSerializer.serialize([1, 2, 3])
    assert str(ei.value) == g["list_type_error"]


def test_oracle_handoff_restatement_matches_reference_serializer(golden):
    from oracle import handoff_ref as H

    g = golden("serializer.json")
    for name, c in g.items():
        if "input_bits_hex" not in c:
            continue
        dt = getattr(torch, c["input_dtype"])
        es = torch.empty((), dtype=dt).element_size()
        raw = np.frombuffer(bytes.fromhex(c["input_bits_hex"]), dtype=np.dtype(f"i{es}")).copy()
        t = torch.from_numpy(raw).view(dt).reshape(c["shape"])
        data, shape, dtype_str = H.wire_bytes(t)
        assert data.hex() == c["bytes_hex"] and list(shape) == c["shape"] and dtype_str == c["dtype_str"], name
        back = H.from_wire(data, shape, dtype_str)
        assert str(back.dtype) == "torch." + c["roundtrip_dtype"]
        got = back.to(torch.float64).flatten().tolist()
        assert all((a == b) or (a != a and b != b) for a, b in zip(got, c["roundtrip_values"])), name
    # a two-layer sequence moved block by block lands in the destination's slots; fp16-representable bf16 is exact
    gen = torch.Generator().manual_seed(5)
    src_k = [torch.randn(6, 2, 16, 8, generator=gen).to(torch.bfloat16) for _ in range(2)]
    src_v = [torch.randn(6, 2, 16, 8, generator=gen).to(torch.bfloat16) for _ in range(2)]
    dst_k = [torch.zeros(5, 2, 16, 8, dtype=torch.bfloat16) for _ in range(2)]
    dst_v = [torch.zeros(5, 2, 16, 8, dtype=torch.bfloat16) for _ in range(2)]
    n = H.handoff_sequence(src_k, src_v, [4, 1, 3], dst_k, dst_v, [0, 2, 1])
    assert n == 2 * 2 * 3 * 2 * 16 * 8 * 2
    for l in range(2):
        assert torch.equal(dst_k[l][[0, 2, 1]], src_k[l][[4, 1, 3]].to(torch.float16).to(torch.bfloat16))
        assert torch.equal(dst_v[l][[0, 2, 1]], src_v[l][[4, 1, 3]].to(torch.float16).to(torch.bfloat16))
        assert not dst_k[l][[3, 4]].any()


def test_streaming_chunks_roundtrip():
    t = torch.arange(3000, dtype=torch.float32).reshape(30, 100)
    data, shape, dt = ser.TensorSerializer.serialize(t)
    tx = ser.StreamingTensorBuffer(chunk_size=1000)
    hdr = tx.write_header(shape, dt)
    rx = ser.StreamingTensorBuffer(chunk_size=1000)
    rx.metadata = rx.read_header(hdr)
    n = 0
    for chunk in tx.iter_chunks(data):
        rx.write_chunk(chunk)
        n += 1
    assert n == 12 and torch.equal(rx.finalize(), t)
    with pytest.raises(ValueError):
        ser.StreamingTensorBuffer().finalize()


# ---- config 1: tiny model, reference ModelShard tokens -----------------------------------------------------
def test_oracle_reproduces_reference_tokens(golden):
    g = golden("tiny_decode.json")
    cfg = L.RefConfig(**g["config"])
    sd = L.make_weights(cfg, seed=0)
    for k, v in g["weights_checksum"].items():
        assert float(sd[k].double().abs().sum()) == pytest.approx(v, rel=1e-12)
    prompts = torch.tensor(g["prompt_ids"])
    assert torch.equal(prompts, torch.randint(0, cfg.vocab_size, (4, 128), generator=torch.Generator().manual_seed(1234)))
    shards = L.build_shards(cfg, sd, [tuple(r) for r in g["shard_ranges"]])
    n = 16  # first 16 of the 64 golden steps keep the CPU suite short
    toks = L.greedy_decode(shards, prompts, n)
    assert toks.tolist() == [row[:n] for row in g["tokens"]]
    assert g["matches_transformers_generate"] is True


def test_oracle_reproduces_reference_tokens_of_the_eight_layer_variant(golden):
    """tiny8_decode.json: eight reference ModelShards of one layer each (what an 8-rank pipeline is checked against)."""
    g = golden("tiny8_decode.json")
    cfg = L.RefConfig(**g["config"])
    assert cfg.num_hidden_layers == 8 and len(g["shard_ranges"]) == 8
    sd = L.make_weights(cfg, seed=0)
    for k, v in g["weights_checksum"].items():
        assert float(sd[k].double().abs().sum()) == pytest.approx(v, rel=1e-12)
    shards = L.build_shards(cfg, sd, [(0, 3), (3, 8)])  # another partition: tokens do not depend on it
    n = 8
    toks = L.greedy_decode(shards, torch.tensor(g["prompt_ids"]), n)
    assert toks.tolist() == [row[:n] for row in g["tokens"]]
    assert g["matches_transformers_generate"] is True


def test_product_seeded_weights_are_the_fixture_weights(golden):
    """dgi_b200.testing.seeded_state_dict (what bench.py's parity check builds its shards from, without touching
    oracle/) draws exactly the weights the golden tokens were generated with."""
    from dgi_b200.testing import LlamaShapeConfig, seeded_state_dict

    for name in ("tiny_decode.json", "tiny8_decode.json"):
        g = golden(name)
        mine = seeded_state_dict(LlamaShapeConfig(**g["config"]), seed=0)
        ref = L.make_weights(L.RefConfig(**g["config"]), seed=0)
        assert list(mine) == list(ref)
        assert all(torch.equal(mine[k], ref[k]) for k in ref)
        for k, v in g["weights_checksum"].items():
            assert float(mine[k].double().abs().sum()) == pytest.approx(v, rel=1e-12)


# ---- paged device ops: oracle == transformers' eager attention, pack == index_select ------------------------
@pytest.mark.parametrize("name", ["float32", "bfloat16", "float16"])
def test_oracle_paged_attention_matches_transformers_eager_golden(golden, name):
    import hashlib

    from oracle import paged_ref as R

    g = golden("paged_ops.json")[name]
    dtype = getattr(torch, name)
    q, k_pool, v_pool, tables, lens = R.golden_case_inputs(dtype)
    raw = lambda x: x.contiguous().view(torch.uint8).numpy().tobytes()  # noqa: E731
    assert hashlib.sha256(raw(q)).hexdigest() == g["q_sha256"]            # the seeded inputs are the fixture's
    assert hashlib.sha256(raw(k_pool)).hexdigest() == g["k_pool_sha256"]
    assert tables.tolist() == g["block_tables"] and lens.tolist() == g["context_lens"]
    eager = R.paged_attention_ref(q, k_pool, v_pool, tables, lens, mode="eager")
    # The committed bytes are transformers' eager_attention_forward as computed on the machine that made the fixture.
    # Another host CPU sums its matmuls in another order, so against the committed bytes the bar is a rounding of the
    # storage dtype ...
    hf = torch.frombuffer(bytearray.fromhex(g["hf_eager_out_hex"]), dtype=dtype).view_as(eager)
    ulp = {"float32": 2e-6, "float16": 2e-3, "bfloat16": 1.6e-2}[name]
    assert (eager.float() - hf.float()).abs().max().item() <= ulp * max(1.0, hf.float().abs().max().item())
    # ... and bit-identity is checked live, on THIS machine, against transformers' own function when it is installed
    try:
        from transformers.models.llama import modeling_llama as hf_llama
    except Exception:  # noqa: BLE001
        hf_llama = None
    if hf_llama is not None:
        from unittest import mock

        B, Hq, D = q.shape
        stub = mock.Mock()
        stub.num_key_value_groups = Hq // k_pool.shape[1]
        stub.training = False
        for b in range(B):
            ctx = int(lens[b])
            if ctx == 0:
                assert not eager[b].any()
                continue
            k = R.gather_dense(k_pool, tables[b], ctx)[None]
            v = R.gather_dense(v_pool, tables[b], ctx)[None]
            o, _ = hf_llama.eager_attention_forward(stub, q[b][None, :, None, :], k, v, None, scaling=D ** -0.5)
            assert torch.equal(o.reshape(Hq, D), eager[b]), f"sequence {b}"
    exact = R.paged_attention_ref(q, k_pool, v_pool, tables, lens, mode="fp32")
    want = torch.frombuffer(bytearray.fromhex(g["exact_fp32_out_hex"]), dtype=torch.float32).view_as(exact)
    assert torch.allclose(exact, want, rtol=0, atol=5e-6)
    packed = R.pack_ref(k_pool, v_pool, torch.tensor(g["packed_seq4_table"], dtype=torch.int32))
    assert hashlib.sha256(raw(packed)).hexdigest() == g["packed_seq4_sha256"]
