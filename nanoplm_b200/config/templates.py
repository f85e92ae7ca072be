"""YAML templates written by `nanoplm pretrain|distill|data get-yaml`.

The key sets are the reference's (src/nanoplm/cli/pretrain.py:594-695, cli/distill.py:540-619,
cli/data.py:676-820) so that files generated by either tool load in the other; keys that only this
framework understands are listed in a separate, commented block of each section.
"""

PRETRAIN_YAML = """\
# Pretraining configuration for nanoplm (B200-native build)
#
# Paths are resolved against the directory you launch from, not against this file.

model:
  hidden_size: 1024
  intermediate_size: 2048
  num_hidden_layers: 16
  num_attention_heads: 16
  vocab_size: 32
  mlp_activation: "swiglu"
  mlp_dropout: 0.0
  mlp_bias: false
  attention_bias: false
  attention_dropout: 0.0
  classifier_activation: "gelu"
  max_position_embeddings: 1024   # must cover the max_seq_len the dataset was prepared with
  # --- optional architecture extensions (all off by default) ---
  # norm_type: "layernorm"        # or "rmsnorm"
  # conv_kernel_size: 0           # 7 = varlen depthwise conv before attention
  # conv_bias: false
  # mhc_streams: 1                # 4 = manifold-constrained hyper-connections
  # mhc_sinkhorn_iters: 5
  # moe:
  #   num_experts: 0              # e.g. 64
  #   top_k: 2
  #   expert_intermediate_size: 512
  #   every_n_layers: 2
  #   aux_loss_coef: 0.01
  #   capacity_factor: 0          # expert parallelism: receive buffers as a multiple of the even share (0 = automatic)

pretraining:
  # Dataset directory: must contain the .data_manifest written by `nanoplm data from-yaml`
  dataset_dir: "output/data/pretrain_shards"

  # Run directories run-DDMMHHMM/ are created below this folder
  ckp_dir: "output/pretraining_checkpoints"

  # Sequences per micro-batch per GPU
  micro_batch_size: 32
  # Tokens per optimizer step over all GPUs; gradient accumulation is derived from
  # global_batch_size / (micro_batch_size * max_seq_len * world_size)
  global_batch_size: 1048576
  num_epochs: 10

  warmup_ratio: 0.05
  optimizer: "adamw"              # adamw | stable_adamw | muon | normuon
  adam_beta1: 0.9
  adam_beta2: 0.999
  adam_epsilon: 1e-8
  adam_learning_rate: 1e-3
  adam_weight_decay: 0.0
  # Used only by muon / normuon (2-D hidden matrices; everything else stays on AdamW)
  muon_learning_rate: 2e-2
  muon_weight_decay: 0.1
  muon_cautious_weight_decay: true
  muon_use_polar_express: false
  muon_momentum: 0.95
  muon_nesterov: true
  muon_eps: 1e-7

  mlm_probability: 0.3
  mask_replace_prob: 0.8
  random_token_prob: 0.1
  keep_probability: 0.1

  logging_steps: 10
  eval_steps: 50
  save_steps: 100
  seed: 42

  num_workers: "auto"
  prefetch_factor: 2

  bf16: true
  tf32: true

  multi_gpu: false
  world_size: 1                   # or "auto" for every visible GPU
  project_name: "nanoplm-pretraining"

  # --- optional extensions ---
  # max_grad_norm: 1.0
  # fp8: false                    # block-scaled e4m3 linears (1x128 activations, 128x128 weights)
  # fp8_recipe: "block128"
  # expert_parallel_size: 1       # ranks per expert-parallel group (must divide the number of ranks)
  # fused_comm: true              # in-kernel reduce-scatter + AdamW + all-gather over NVLink
  # sharded_checkpoint: false
  # device_masking: false
  # metrics_jsonl: true
  # heartbeat_seconds: 0
  # heartbeat_stall_seconds: 0    # > 0: end the job when a rank makes no progress for this long
  # balance_ranks: true           # equal-cost micro-batches on every rank (static packing, several GPUs)
  # shard_params: false           # shard the layers' weights over the ranks (all-gather fused into the GEMMs)
  # nvtx_ranges: false            # NVTX ranges around forward / backward / optimizer step
  # deterministic_attention: false  # attention backward and linear weight gradients bitwise reproducible (slower)
  # hf_checkpoint_files: false    # also write model.safetensors + trainer_state.json with every checkpoint

# The native pipeline (own CUDA kernels, sharded data parallelism). `use_compile` is accepted for
# compatibility and ignored; packing removes padding, target_packed_rows fixes the flat length.
pure_torch:
  enabled: true
  use_compile: true
  use_packing: true
  target_packed_rows: null

resume:
  is_resume: false
  checkpoint_dir: "output/pretraining_checkpoints/run-1/checkpoint-1"
  extra_epochs: 0
"""

DISTILL_YAML = """\
# Distillation configuration for nanoplm (B200-native build)
#
# Paths are resolved against the directory you launch from, not against this file.

model:
  hidden_size: 512
  intermediate_size: 1024
  num_hidden_layers: 6
  num_attention_heads: 8
  mlp_activation: "swiglu"
  mlp_dropout: 0.0
  mlp_bias: false
  attention_bias: false
  attention_dropout: 0.0
  classifier_activation: "gelu"
  projection_layer: true          # project the student width to the teacher's 1024
  # --- optional architecture extensions ---
  # conv_kernel_size: 0
  # mhc_streams: 1
  # norm_type: "layernorm"

distillation:
  # Dataset directory: must contain the .data_manifest written by `nanoplm data from-yaml`
  dataset_dir: "output/data/kd_dataset"
  ckp_dir: "output/distillation_checkpoints"

  num_epochs: 10
  batch_size: 64
  learning_rate: 1e-3
  gradient_accumulation_steps: 1
  warmup_ratio: 0.05

  lr_scheduler: "cosine"          # cosine | linear | polynomial | constant
  lr_scheduler_kwargs: {}

  # Pre-computed (HDF5) datasets
  max_open_files: 5
  chunk_size: 32
  prefetch_batches: 2
  use_threading: true
  num_workers: 8

  project_name: "nanoplm-distillation"
  logging_steps: 10
  eval_steps: 50
  save_steps: 100

  bf16: true
  tf32: true

  multi_gpu: false
  world_size: 1
  seed: 42

  # --- optional extensions ---
  # teacher_random_init: false    # frozen random-init teacher (benchmarks, offline machines)
  # heartbeat_seconds: 0          # > 0: per-rank heartbeat files under <run>/heartbeat (see `distill supervise`)
  # heartbeat_stall_seconds: 0    # > 0: end the job when a rank makes no progress for this long
  # teacher: {d_model: 1024, d_ff: 16384, num_layers: 24, num_heads: 32, d_kv: 128, vocab_size: 128}

resume:
  is_resume: false
  checkpoint_dir: "output/distillation_checkpoints/run-1/checkpoint-1"
  extra_epochs: 0
"""

PARAMS_YAML = """\
# Data preparation parameters for nanoplm (consumed by dvc.yaml and `nanoplm data from-yaml`)

data_params:
  pipeline_mode: "pretrain"       # none | pretrain | distillation
  seqs_num: 20000                 # -1 keeps every sequence that passes the length filter
  min_seq_len: 20
  max_seq_len: 512
  val_ratio: 0.1
  device: "auto"
  shuffle_backend: "biopython"    # biopython (in-process) | seqkit (external binary)
  shuffle: true
  shuffle_seed: 24
  filter_skip_n: 0

pretrain_config:
  output_dir: "output/data/pretrain_shards"
  samples_per_shard: 2000
  max_workers: 2                  # -1 = all cores
  force: false

distillation_config:
  output_dir: "output/data/kd_dataset"
  on_the_fly: false
  samples_per_shard: 2000         # -1 = one file
  teacher_model: "prott5"
  embed_calc_batch_size: 4

data_dirs:
  url: "https://ftp.uniprot.org/pub/databases/uniprot/current_release/knowledgebase/complete/uniprot_sprot.fasta.gz"
  compressed_fasta: "output/data/raw/uniref50.fasta.gz"
  extracted_fasta: "output/data/raw/uniref50.fasta"
  shuffled_fasta: "output/data/raw/uniref50_shuffled.fasta"
  filtered_fasta: "output/data/filter/uniref50_filtered.fasta"
  splitted_fasta_dir: "output/data/split"
"""

DVC_YAML = """\
# DVC pipeline for nanoplm data preparation. Every stage is one `nanoplm data ...` command.
stages:
  download:
    cmd: nanoplm data download --url ${data_dirs.url} -o ${data_dirs.compressed_fasta} --force
    params:
      - data_dirs.url
    outs:
      - ${data_dirs.compressed_fasta}

  extract:
    cmd: nanoplm data extract -i ${data_dirs.compressed_fasta} -o ${data_dirs.extracted_fasta} --force
    deps:
      - ${data_dirs.compressed_fasta}
    outs:
      - ${data_dirs.extracted_fasta}

  shuffle:
    cmd: nanoplm data shuffle -i ${data_dirs.extracted_fasta} -o ${data_dirs.shuffled_fasta} --backend ${data_params.shuffle_backend} --seed ${data_params.shuffle_seed}
    deps:
      - ${data_dirs.extracted_fasta}
    params:
      - data_params.shuffle_backend
      - data_params.shuffle_seed
    outs:
      - ${data_dirs.shuffled_fasta}

  filter:
    cmd: nanoplm data filter -i ${data_dirs.shuffled_fasta} -o ${data_dirs.filtered_fasta} --min-seq-len ${data_params.min_seq_len} --max-seq-len ${data_params.max_seq_len} --seqs-num ${data_params.seqs_num} --skip-n ${data_params.filter_skip_n}
    deps:
      - ${data_dirs.shuffled_fasta}
    params:
      - data_params.min_seq_len
      - data_params.max_seq_len
      - data_params.seqs_num
      - data_params.filter_skip_n
    outs:
      - ${data_dirs.filtered_fasta}

  split:
    cmd: nanoplm data split -i ${data_dirs.filtered_fasta} -o ${data_dirs.splitted_fasta_dir} --val-ratio ${data_params.val_ratio}
    deps:
      - ${data_dirs.filtered_fasta}
    params:
      - data_params.val_ratio
    outs:
      - ${data_dirs.splitted_fasta_dir}/train.fasta
      - ${data_dirs.splitted_fasta_dir}/val.fasta

  save_kd_train_dataset:
    cmd: nanoplm data save-kd-dataset -i ${data_dirs.splitted_fasta_dir}/train.fasta -o ${distillation_config.output_dir}/train/train_kd_dataset.h5 --teacher-model ${distillation_config.teacher_model} --max-seq-len ${data_params.max_seq_len} --batch-size ${distillation_config.embed_calc_batch_size} --device ${data_params.device} --samples-per-shard ${distillation_config.samples_per_shard} --force
    deps:
      - ${data_dirs.splitted_fasta_dir}/train.fasta
    params:
      - distillation_config.teacher_model
      - distillation_config.samples_per_shard
      - data_params.max_seq_len
    outs:
      - ${distillation_config.output_dir}/train

  save_kd_val_dataset:
    cmd: nanoplm data save-kd-dataset -i ${data_dirs.splitted_fasta_dir}/val.fasta -o ${distillation_config.output_dir}/val/val_kd_dataset.h5 --teacher-model ${distillation_config.teacher_model} --max-seq-len ${data_params.max_seq_len} --batch-size ${distillation_config.embed_calc_batch_size} --device ${data_params.device} --samples-per-shard ${distillation_config.samples_per_shard} --force
    deps:
      - ${data_dirs.splitted_fasta_dir}/val.fasta
    params:
      - distillation_config.teacher_model
      - distillation_config.samples_per_shard
      - data_params.max_seq_len
    outs:
      - ${distillation_config.output_dir}/val
"""
