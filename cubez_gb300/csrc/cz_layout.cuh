// Device layout of a batch of independent worlds (structure of arrays).
//
// Bodies: one row per field, each row `nb_pad` long; world w owns rows
// [body_start[w], body_start[w] + body_count[w]) with body_start a multiple of
// 4, so that every world's slice of a row starts on a 16-byte (float) or
// 32-byte (double) boundary and can be staged with a bulk copy.
// Contacts: one row per field, each `nc_total` long; world w owns
// [contact_start[w], contact_start[w] + contact_cap[w]).
#pragma once
#include <cstdint>

#include "cz_mlp.cuh"

namespace cz {

// integer rows of the per-body warm-start scratch
enum WsInt : int {
  WS_DEG = 0,   // contacts touching the body
  WS_NBB,       // contacts between the body and other bodies
  WS_LOAD,      // sum of their positive desired delta velocities, fixed point 2^-16
  WS_FIRST,     // first and last index of the body's half-space contacts
  WS_LAST,
  WS_SCALE,     // warm-start scale (float bits)
  WS_NINT
};
constexpr float kLoadScale = 65536.f;

enum BodyRow : int {
  B_PX, B_PY, B_PZ,                                      // RigidBody.Position
  B_QW, B_QX, B_QY, B_QZ,                                // RigidBody.Orientation
  B_HX, B_HY, B_HZ, B_RAD,                               // CollisionCube.HalfSize / CollisionSphere.Radius
  B_VX, B_VY, B_VZ,                                      // Velocity
  B_RX, B_RY, B_RZ,                                      // Rotation (angular velocity)
  B_AX, B_AY, B_AZ,                                      // Acceleration
  B_LX, B_LY, B_LZ,                                      // lastFrameAccelleration
  B_IB0, B_IB1, B_IB2, B_IB3, B_IB4, B_IB5, B_IB6, B_IB7, B_IB8,  // InverseInertiaTensor (body)
  B_IW0, B_IW1, B_IW2, B_IW3, B_IW4, B_IW5, B_IW6, B_IW7, B_IW8,  // inverseInertiaTensorWorld
  B_INVM,                                                // inverseMass
  B_LINPOW, B_ANGPOW,                                    // pow(LinearDamping, dt), pow(AngularDamping, dt)
  B_MOTION,                                              // motion
  B_NROWS
};

// Narrowphase output (Contact fields set by the colliders).
enum ContactRow : int { C_PX, C_PY, C_PZ, C_NX, C_NY, C_NZ, C_PEN, C_FRIC, C_REST, C_NROWS };

// Resolver working set (Contact's private fields, contact.go:38-50): one
// record of CREC reals per contact, read in 16-byte pieces.  The basis's second
// and third columns are functions of the normal (calculateContactBasis,
// contact.go:114-156); they are kept, as recomputing them where the basis is
// used costs more instructions than their loads.
enum ContactRec : int {
  CR_N = 0,     // contactToWorld's columns: normal,
  CR_TY = 3,    //   tangent y,
  CR_TZ = 6,    //   tangent z
  CR_R0 = 9,    // relative contact positions
  CR_R1 = 12,
  CR_PEN = 15,  // penetration (adjustPositions); then
  CR_VFA = 15,  // the frame velocity along the normal (adjustVelocities)
  CR_CV = 16,   // contact velocity
  CR_DDV = 19,  // desired delta velocity
  CREC = 20
};
// Working state of a body, one record of BREC reals (position and orientation
// are kept apart, in the island type)
enum BodyRec : int { BR_VEL = 0, BR_ROT = 3, BR_IIT = 6, BR_INVM = 15, BR_LFA = 16, BR_MOTION = 19, BREC = 20 };
// reals per contact of the friction solve's matrices (K: 9, the response's
// first row: 3, padding: 4), contact-major, so the resolved contact's are one
// aligned 64- (float32) or 128-byte (float64) block
constexpr int K_ROW = 16;

// World status bits (also OR-ed into the batch status word).
enum : uint32_t {
  ST_NONFINITE = 1u,        // box-box test reached with no accepted axis (non-finite state)
  ST_FRICTIONLESS_NIL = 2u, // frictionless impulse on a single-body contact (the reference panics)
  ST_CAPACITY = 4u,         // more contacts than the world's capacity
  ST_TIMEOUT = 8u,          // a bounded wait gave up
  ST_BODY_LIMIT = 16u,      // world larger than the kernel's shared-memory tile
};

// in BatchView::cost: the world's last adjustVelocities used its whole budget
constexpr int kExhausted = 1 << 30;
// Worlds of more bodies than this list more units for the narrowphase than a
// chunk or two of its CTA hold (np_flush).
constexpr int kPairedBodies = 64;
// k_narrowphase's instantiation for a batch: worlds of up to kPairedBodies
// bodies, larger ones, or with the grid
enum NPMode { NP_SMALL, NP_LARGE, NP_GRID };
inline NPMode np_mode(int grid_min_bodies, int max_bodies) {
  if (grid_min_bodies > 0 && max_bodies >= grid_min_bodies) return NP_GRID;
  return max_bodies > kPairedBodies ? NP_LARGE : NP_SMALL;
}

// packed body pair of a contact: low 16 bits body 0, high 16 bits body 1
// (0xFFFF = nil).  World-local indices, so a world holds at most 65535 bodies.
__host__ __device__ __forceinline__ int pack_bodies(int b0, int b1) {
  return (int)(((unsigned)(b0 & 0xFFFF)) | ((unsigned)(b1 & 0xFFFF) << 16));
}
__host__ __device__ __forceinline__ int body0_of(int p) {
  int b = p & 0xFFFF;
  return b == 0xFFFF ? -1 : b;
}
__host__ __device__ __forceinline__ int body1_of(int p) {
  int b = (int)(((unsigned)p) >> 16);
  return b == 0xFFFF ? -1 : b;
}

template <class R> struct BatchView {
  R* body;              // [B_NROWS][nb_pad]
  uint8_t* awake;       // [nb_pad]
  uint8_t* can_sleep;   // [nb_pad]
  int32_t* shape;       // [nb_pad] 0 sphere, 1 cube, -1 padding
  const R* offset;      // [12][nb_pad] collider Offset (column-major 3x4), null = identity for every body
  long long nb_pad;
  // the worlds a launch covers: num_worlds of them from first_world, whose
  // bodies are the nb_run padded rows from first_body
  long long first_body, nb_run;
  int first_world;
  int num_worlds;
  int max_bodies;       // largest world
  const int* body_start;
  const int* body_count;
  const long long* contact_start;
  const int* contact_cap;
  int* contact_count;   // [num_worlds] narrowphase output
  uint32_t* world_status;
  int* pos_iters;
  int* vel_iters;
  int* cost;            // [num_worlds] the resolver's rounds in the last frame (k_reorder), and kExhausted
  R* contact;           // [C_NROWS][nc_total]
  int* contact_bodies;  // [nc_total]
  R* work;              // [nc_total][CREC] contact records of the worlds above the shared tile
  R* kmat;              // [nc_total][16] reals per contact: K of its friction solve (9, inverted in the
                        // island type), the friction response's first row (3), padding (4)
  int* work_bodies;     // [nc_total]
  long long nc_total;
  const int* order;     // narrowphase queue: worlds in decreasing body count
  const int* order_rs;  // resolver queue: worlds in decreasing iterations of the previous frame
  unsigned* queue;      // [0] narrowphase, [1] resolver, [2] features, [3] spare (k_integrate zeroes them)
  uint32_t* status;     // batch status word
  unsigned long long* counters;  // [0] contacts generated, [1] adjustPositions iterations,
                                 // [2] adjustVelocities iterations, [3] contacts resolved,
                                 // [4] warm-started worlds re-solved plainly, [5] warm-started worlds
  R plane_nx, plane_ny, plane_nz, plane_offset;
  int iter_mult;        // ResolveContacts(len(contacts) * iter_mult)
  int max_iterations;   // >= 0 overrides len(contacts) * iter_mult
  int contact_writeback; // copy the resolved contacts back to the contact rows
  int uniform_material;  // every contact has the colliders' friction 0.9 / restitution 0.1
  int mode;              // resolver: 0 plain, 1 harvest, 2 learned warm start
  MlpDev mlp;            // warm-start network (mode 2)
  float* hv_features;    // harvest output [hv_cap][18]
  float* hv_labels;      // harvest output [hv_cap][3]
  unsigned long long* hv_count;
  long long hv_cap;
  // per-body scratch of the warm start and the harvest (modes 1, 2), indexed
  // like the body rows (row stride nb_pad)
  R* ws_rows;            // [6]: warm-start velocity and rotation change
  R* ws_imp;             // [3][nc_total] contact-frame impulse: predicted (warm start) or applied in total (harvest)
  int* ws_int;           // [WS_NINT]
  uint8_t* ws_world;     // [num_worlds]: the world's last velocity solve used more than max_it >> warm_shift
  float* ws_feat;        // [nc_total][18] harvest features (k_warm_features, mode 1)
  int warm_shift;        // warm-start a world when its last solve used <= max_it >> warm_shift
  // worlds above the shared-memory slot of k_resolve, resolved by k_resolve_big
  const int* big_list;   // [big_count] world ids
  int big_count;
  void* big_bw;          // [nb_pad][7] positions / orientations in the island type
  R* big_br;             // [nb_pad][BREC] body records
  uint8_t* big_aw;       // [nb_pad] awake flags
  // of worlds whose contacts exceed k_resolve_big's shared memory:
  int* big_adj;          // [2 * nc_total] contact lists per body, a world's segment at 2 * contact_start
  void* big_key;         // [nc_total] argmax keys (as wide as R)
  // the narrowphase's bounded wait on its staging copies: polls before it
  // gives up, and extra bytes expected beyond those copied (0; a test raises
  // it so that the wait runs out with every real copy landed)
  int wait_limit;
  int wait_extra_tx;
  int grid_min_bodies;  // narrowphase: worlds of at least this many bodies use the grid (0: none)
};

}  // namespace cz
